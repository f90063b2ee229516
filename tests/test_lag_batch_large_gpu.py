"""Lagrangian batches on both sides of the line between the cell kernels (28,000 cells of the
table): a table above it, with problems that leave part of a tile empty, and one that
problems take across it in both directions. Each problem ends with its solo result, bit for
bit, and the step loop is captured once for either side."""
import numpy as np
import pytest

from test_lag_batch_gpu import _problem, _solo

pytestmark = pytest.mark.gpu


def _slab(nx, ny, seed):
    from subfv_b200 import meshgen
    return meshgen.prism_slab(nx, ny, 0.0, 1.2, 0.0, 1.2, 0.0, 0.1, jitter=0.05, seed=seed)


def _same(batch, k, m, raw, cfl, t_max, steps, precision):
    st, n, t, ref, x = _solo(raw, cfl, t_max, steps, precision)
    bt, bn, _, bst = batch.info(k)
    assert (bst, bn, bt) == (st, n, t) and st == 0
    np.testing.assert_array_equal(batch.sol(k, m.n_elems), ref)
    np.testing.assert_array_equal(m.coords(), x)


@pytest.mark.parametrize("precision", [0, 1])
def test_large_table(native, cuda_ok, precision):
    from subfv_b200 import meshgen
    from subfv_b200.lagrange import LagBatch
    cases = [(_slab(101, 99, 3), 0.5, 1.0), (_slab(61, 57, 4), 0.4, 1.0), (_slab(5, 7, 5), 0.3, 0.2),
             (meshgen.hex_slab(37, 41, 0.0, 1.2, 0.0, 1.2, 0.0, 0.1, jitter=0.05, seed=6), 0.5, 0.05)]
    b = LagBatch(capacity=8, budget_bytes=1 << 34, precision=precision)
    probs = []
    for raw, cfl, t_max in cases:
        m, sol = _problem(raw)
        probs.append((m, b.add(m, sol, t_max, cfl=cfl)))
    assert sum(m.n_elems for m, _ in probs) > 28000
    b.advance(16)
    b.advance(5)
    b.sync()
    for (raw, cfl, t_max), (m, k) in zip(cases, probs):
        _same(b, k, m, raw, cfl, t_max, 21, precision)
    b.close()


def test_table_crosses_the_line(native, cuda_ok):
    from subfv_b200 import _lib
    from subfv_b200.lagrange import LagBatch
    captures = _lib.load().subfv_probe_lag_captures
    big, other = _slab(110, 100, 7), _slab(57, 55, 8)
    b = LagBatch(capacity=4, budget_bytes=1 << 34)
    m, sol = _problem(big)
    k = b.add(m, sol, 1.0, cfl=0.5)
    b.advance(8)
    steps = 8
    for _ in range(3):
        m2, sol2 = _problem(other)
        k2 = b.add(m2, sol2, 1.0, cfl=0.5)
        b.advance(11)
        b.sync()
        _same(b, k2, m2, other, 0.5, 1.0, 11, 0)
        b.remove(k2)
        b.advance(9)
        steps += 20
    b.sync()
    _same(b, k, m, big, 0.5, 1.0, steps, 0)
    assert captures(b._h) == 2
    b.close()
