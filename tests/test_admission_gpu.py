"""Admitting a problem to a batch does not wait for the work queued on its mesh's stream."""
import ctypes
import threading
import time

import numpy as np
import pytest

from test_ns_gpu import _perturbed_gresho

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", [1, 4, 5])
@pytest.mark.parametrize("second_order", [False, True])
def test_admission_does_not_wait(native, cuda_ok, scheme, second_order):
    from subfv_b200 import meshgen
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsBatch, NsConfig, NsState
    cfg = NsConfig(scheme=scheme, second_order=second_order, method=4, bc_style=2, boundary_2d=True, cfl=0.4)
    first, m = (Mesh.from_raw(meshgen.hex_slab(9, 7, jitter=0.1, seed=i)) for i in (3, 4))
    sol = _perturbed_gresho(m, 5)
    b = NsBatch(cfg, capacity=4, budget_bytes=1 << 30)
    assert b.add(first, _perturbed_gresho(first, 5), 1e30) is not None  # the kernels are loaded
    b.advance(1)
    b.sync()
    go = threading.Event()
    hold = ctypes.CFUNCTYPE(None, ctypes.c_void_p)(lambda _: go.wait(3.0) and None)
    rt = ctypes.CDLL("libcudart.so.12")
    native.subfv_mesh_stream.restype = ctypes.c_void_p
    assert rt.cudaLaunchHostFunc(ctypes.c_void_p(native.subfv_mesh_stream(m._h)), hold, None) == 0
    t0 = time.perf_counter()
    k = b.add(m, sol, 1e30)
    took = time.perf_counter() - t0
    go.set()
    assert k is not None and took < 1.5, took
    b.advance(6)
    b.sync()
    s = NsState(m, cfg, sol)
    st, n, t = s.advance(6)
    assert b.info(k)[:2] == (t, n) and st == 0
    np.testing.assert_array_equal(b.sol(k, m.n_elems), s.sol())
    b.close()
