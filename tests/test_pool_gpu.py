"""The pool that states and batch slots allocate from: freed memory is kept for the next one
however much is in use, and all but 512 MB (in steps of 64 MB) is given back once it is no
longer in use."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free_bytes():
    rt = ctypes.CDLL("libcudart.so.12")
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    assert rt.cudaDeviceSynchronize() == 0
    assert rt.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def test_pool_keeps_beyond_its_use_and_gives_back(native, cuda_ok):
    from subfv_b200 import meshgen
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsConfig, NsState
    m = Mesh.from_raw(meshgen.hex_slab(300, 300, jitter=0.0, seed=0))
    cfg = NsConfig(scheme=1, second_order=False, method=0, bc_style=2, boundary_2d=True, cfl=0.4)
    sol = np.zeros((m.n_elems, 5))
    sol[:, 0], sol[:, 4] = 1.0, 2.5
    first = NsState(m, cfg, sol)  # what the mesh and the pool set up once
    first.close()
    start = _free_bytes()
    live = [NsState(m, cfg, sol) for _ in range(16)]
    in_use = start - _free_bytes()
    assert in_use > 600 * MB  # past what the pool keeps
    size = in_use // 16
    s = NsState(m, cfg, sol)
    s.close()
    live[0].sol()  # synchronises the mesh's stream
    kept = start - _free_bytes() - in_use
    assert kept >= size // 2
    for _ in range(3):  # the next state takes it: no growth
        s = NsState(m, cfg, sol)
        s.close()
        live[0].sol()
    assert start - _free_bytes() - in_use <= kept
    for x in live:
        x.close()
    m.coords()
    _free_bytes()
    assert start - _free_bytes() <= (512 + 2 * 64) * MB
