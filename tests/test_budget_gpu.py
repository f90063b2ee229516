"""What a batch's budget admits: a problem is charged its mesh and its state records, not the
caches that faster kernels keep with the mesh; with room for no more than the charge it is
admitted, runs without them and ends with its solo state."""
from dataclasses import replace

import numpy as np
import pytest

from test_ns_gpu import _perturbed_gresho

pytestmark = pytest.mark.gpu


def _raw(name):
    from subfv_b200 import meshgen
    return {"quads": lambda: meshgen.hex_slab(13, 9, jitter=0.1, seed=3),
            "tris": lambda: meshgen.prism_slab(9, 8, -0.5, 0.5, -0.5, 0.5, -0.5, 0.5, jitter=0.05, seed=4),
            "strip": lambda: meshgen.strip(57),
            "box": lambda: meshgen.hex_box(4, jitter=0.05, seed=5, periodic=True)}[name]()


@pytest.mark.parametrize("second_order", [False, True])
@pytest.mark.parametrize("scheme", [1, 4, 5])
@pytest.mark.parametrize("name", ["quads", "tris", "strip", "box"])
def test_budget_admits_by_mesh_and_records(native, cuda_ok, name, scheme, second_order):
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsBatch, NsConfig, NsState
    m = Mesh.from_raw(_raw(name))
    ne, nv, nse = m.n_elems, m.n_vert, len(m.topo.array("sub_elem_vert"))
    blocks = -(-ne // 128)
    records = 8 * (8 * ne + 6 * nse + 6 * ne + 5 * ne + 6 * blocks)
    if second_order:
        records += 8 * (8 * ne + 6 * ne + 15 * nv + 15 * ne)
    cfg = NsConfig(scheme=scheme, second_order=second_order, method=4, bc_style=2, boundary_2d=name != "box", cfl=0.4)
    sol = _perturbed_gresho(m, 5)
    need = records + m.device_bytes
    got = []
    for budget in (need, 1 << 30, need):  # the caches are built in between
        b = NsBatch(cfg, capacity=2, budget_bytes=budget)
        assert b.state_bytes(m) == records
        k = b.add(m, sol, 1e30)
        assert k is not None and b.free_bytes() == budget - need
        b.advance(9)
        b.sync()
        got.append((b.info(k), b.sol(k, ne)))
        b.close()
    other = Mesh.from_raw(_raw(name))
    b = NsBatch(cfg, capacity=2, budget_bytes=need - 1)
    assert b.add(other, sol, 1e30) is None
    b.close()
    s = NsState(m, replace(cfg, tmax=1e30), sol)
    st, n, t = s.advance(9)
    for (bt, bn, _, bst), x in got:
        assert (bst, bn, bt) == (st, n, t)
        np.testing.assert_array_equal(x, s.sol())
