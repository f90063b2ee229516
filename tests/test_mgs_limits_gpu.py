"""The one-launch Gram-Schmidt column against its limits. Where its grid may not be resident
one launch per projection serves; on one or two blocks the elements beyond the registers
fill shared memory row by row (27 rows at most), and a vector beyond those takes one launch
per projection again. H as in test_mgs_column_gpu.py: n terms round by less than
n 2^-53 |w| |v| <= 1e-11 |w| |v| at these sizes, and |w| is at most the operator's norm, 4."""
import numpy as np
import pytest

from test_mgs_column_gpu import _arnoldi

pytestmark = pytest.mark.gpu


def _tridiagonal(n):
    from subfv_b200.bcsr import BcsrMatrix, DeviceBcsr
    rng = np.random.default_rng(n)
    d, l, u = rng.uniform(1, 2, n), rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    i = np.arange(n)
    col = np.stack([i - 1, i, i + 1], 1).ravel()
    keep = (col >= 0) & (col < n)
    row = np.concatenate([[0], np.cumsum(keep.reshape(n, 3).sum(1))])
    A = DeviceBcsr(BcsrMatrix(n, 1, (row + 1).astype(np.int32), (col[keep] + 1).astype(np.int32),
                              np.stack([l, d, u], 1).ravel()[keep].reshape(-1, 1, 1)))

    def mul(x):
        y = d * x
        y[1:] += l[1:] * x[:-1]
        y[:-1] += u[:-1] * x[1:]
        return y

    return A, mul, rng.standard_normal(n)


def _limit(A, blocks, polls=0):
    from subfv_b200 import _lib
    _lib.check(_lib.load().subfv_probe_gram_schmidt(A._h, blocks, polls), "subfv_probe_gram_schmidt")


@pytest.mark.parametrize("blocks, n", [(0, 1), (0, 5000), (1, 1024), (1, 8 * 1024 + 1), (1, 17 * 1024), (1, 20 * 1024 + 3),
                                       (1, 43 * 1024 - 1), (1, 43 * 1024), (1, 43 * 1024 + 1), (2, 38 * 1024 + 7)])
def test_gram_schmidt_with_fewer_blocks(native, cuda_ok, blocks, n):
    A, mul, b = _tridiagonal(n)
    m = min(5, n)
    _limit(A, blocks)
    *_, H = A.gmres(b, 1e-300, m, precond=False, want_h=True)
    if n > m:
        np.testing.assert_allclose(H.T, _arnoldi(mul, b, m), rtol=0, atol=4 * 1e-11)
    else:
        np.testing.assert_allclose(H[0, 0], mul(np.ones(n))[0], rtol=1e-14)


@pytest.mark.parametrize("flush", [False, True])
def test_wait_that_runs_out_is_an_error(native, cuda_ok, flush):
    """Blocks that give up after one poll (an answer takes several times as long) make the
    solve return an error, also in a process that flushes subnormals to zero; the next solve
    on the handle is sound."""
    import torch
    A, mul, b = _tridiagonal(5000)
    _limit(A, -1, polls=1)
    assert torch.set_flush_denormal(flush)
    try:
        with pytest.raises(RuntimeError, match="waited too long"):
            A.gmres(b, 1e-300, 5, precond=False)
    finally:
        torch.set_flush_denormal(False)
    _limit(A, -1)
    *_, H = A.gmres(b, 1e-300, 5, precond=False, want_h=True)
    np.testing.assert_allclose(H.T, _arnoldi(mul, b, 5), rtol=0, atol=4 * 1e-11)
