"""The one-launch Gram-Schmidt column at the edges of its layouts: vectors of one element, of
one block and one more, and of one more element than the registers of 1, 2, 4, 8 and 16 per
thread hold on 148 SMs (the last spills into shared memory). H against a modified
Gram-Schmidt in numpy: each entry is a dot product of n terms whose rounding is below
n 2^-53 |w| |v| <= 3e-10 |w| |v|, and |w| is at most the operator's norm, 4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T = 148 * 1024


def _arnoldi(mul, b, m):
    V, H = [b / np.linalg.norm(b)], np.zeros((m + 1, m))
    for j in range(m):
        w = mul(V[j])
        for i in range(j + 1):
            H[i, j] = w @ V[i]
            w = w - H[i, j] * V[i]
        H[j + 1, j] = np.linalg.norm(w)
        V.append(w / H[j + 1, j])
    return H


@pytest.mark.parametrize("n", [7, 1023, 1024, 1025, T, T + 1, 2 * T + 1, 4 * T + 1, 8 * T + 1, 16 * T + 1])
def test_gram_schmidt_column(native, cuda_ok, n):
    from subfv_b200.bcsr import BcsrMatrix, DeviceBcsr
    rng = np.random.default_rng(n)
    m = 5
    d, l, u = rng.uniform(1, 2, n), rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)  # tridiagonal
    row = np.concatenate([[0], np.cumsum(np.where((np.arange(n) == 0) | (np.arange(n) == n - 1), 2, 3))])
    i = np.arange(n)
    col = np.stack([i - 1, i, i + 1], 1).ravel()
    val = np.stack([l, d, u], 1).ravel()
    keep = (col >= 0) & (col < n)
    A = DeviceBcsr(BcsrMatrix(n, 1, (row + 1).astype(np.int32), (col[keep] + 1).astype(np.int32),
                              val[keep].reshape(-1, 1, 1)))

    def mul(x):
        y = d * x
        y[1:] += l[1:] * x[:-1]
        y[:-1] += u[:-1] * x[1:]
        return y

    b = rng.standard_normal(n)
    *_, H = A.gmres(b, 1e-300, m, precond=False, want_h=True)
    np.testing.assert_allclose(H.T, _arnoldi(mul, b, m), rtol=0, atol=4 * 3e-10)
