"""Coordinates and states are read and set on the device that holds them, whichever device is
current, and the caller's device stays current. Needs a second device."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_reads_with_another_device_current(native, cuda_ok):
    if cuda_ok < 2:
        pytest.skip("one device")
    from subfv_b200 import meshgen
    from subfv_b200.lagrange import LagBatch, LagrangeState, init_sol_sedov
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsConfig, NsState, init_gresho
    rt = ctypes.CDLL("libcudart.so.12")
    cur = ctypes.c_int()

    def read(m, s, lag, batch, k, lm):
        return [m.coords(), s.sol(), lag.vp(), batch.sol(k, lm.n_elems), lm.coords()]

    m, lm, bm = (Mesh.from_raw(meshgen.prism_slab(12, 10, jitter=0.05, seed=i)) for i in (1, 2, 3))
    s = NsState(m, NsConfig(cfl=0.4), init_gresho(m, 0.1))
    sol = init_sol_sedov(lm, e_total=0.1)
    lag = LagrangeState(lm, sol, cfl=0.5, t_max=1.0)
    batch = LagBatch(capacity=2, budget_bytes=1 << 30)
    k = batch.add(bm, init_sol_sedov(bm, e_total=0.1), 1.0, cfl=0.5)
    s.advance(2), lag.advance(2), batch.advance(2), batch.sync()
    ref = read(m, s, lag, batch, k, bm)
    assert rt.cudaSetDevice(1) == 0
    try:
        got = read(m, s, lag, batch, k, bm)
        m.set_coords(ref[0])
        assert rt.cudaGetDevice(ctypes.byref(cur)) == 0 and cur.value == 1
    finally:
        rt.cudaSetDevice(0)
    for a, b in zip(ref, got):
        np.testing.assert_array_equal(a, b)
