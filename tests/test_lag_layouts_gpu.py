"""The Lagrangian step on both sides of the lines between its cell kernels, bit for bit
against the oracle: the last mesh of the tile kernels and the first of the thread-per-cell
ones (28,000 cells), and the thread-per-cell geometry's two splits of shared memory (up to
7 blocks of 64 cells an SM, between 7 and 10, above 10)."""
import numpy as np
import pytest

from test_lagrange_gpu import _pair, _sedov

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, ny", [(125, 112), (127, 111), (188, 179), (225, 212)])
def test_cell_kernels_bit_exact(native, oracle_lib, cuda_ok, nx, ny):
    from subfv_b200 import meshgen
    from subfv_b200.lagrange import LagrangeState
    m, o = _pair(meshgen.prism_slab(nx, ny, jitter=0.05, seed=3))
    sol = _sedov(m, o)
    mass = m.geometry("elem_volume") / sol[:, 0]
    s = LagrangeState(m, sol, mass, cfl=0.8, t_max=1.0)
    assert s.run(max_steps=3)[:2] == (0, 3)
    sol_o = sol.copy()
    o.lag_run(sol_o, mass, 0.8, 1.0, 3)
    np.testing.assert_array_equal(s.sol(), sol_o)
    np.testing.assert_array_equal(m.coords(), o.geom("vert_coord"))
    for name in ("elem_volume", "elem_coord", "sub_elem_volume"):
        a, b = m.geometry(name), o.geom(name)
        np.testing.assert_array_equal(a.reshape(b.shape), b, err_msg=name)
