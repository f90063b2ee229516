"""The Lagrangian arrays' charge to a mesh: the face records, the entries of the cells' lists,
16 bytes of codes a cell and 4 a subcell, whatever the tiles they lie in take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def wedge():
    """A hexahedron with a prism on its x side: cells of 24 and 18 entries."""
    from subfv_b200 import meshgen
    xy = np.array([[0, 0], [1, 0], [1, 1], [0, 1], [1.8, 0.5]], float)
    coords = np.column_stack([np.tile(xy, (2, 1)), np.repeat([0.0, 1.0], 5)])
    ev = [0, 1, 2, 3, 5, 6, 7, 8] + [1, 4, 2, 6, 9, 7]
    return meshgen.RawMesh(coords, np.array([meshgen.KIND_HEX, meshgen.KIND_PRISM], np.int32),
                           np.array([0, 8, 14], np.int32), np.array(ev, np.int32) + 1, b2d=True)


@pytest.mark.parametrize("name", ["tris", "quads", "wedge"])
def test_lagrangian_arrays_charge(native, cuda_ok, name):
    from subfv_b200 import meshgen
    from subfv_b200.lagrange import LagBatch
    from subfv_b200.mesh import Mesh
    raw = {"tris": lambda: meshgen.prism_slab(9, 7, jitter=0.05, seed=1),
           "quads": lambda: meshgen.hex_slab(7, 5, 0.0, 1.2, 0.0, 1.2, 0.0, 0.1, jitter=0.05, seed=1),
           "wedge": wedge}[name]()
    m = Mesh.from_raw(raw)
    t = m.topo
    left, right, face = t.array("face_left"), t.array("face_right"), t.array("sub_face_face")
    entries = len(face) + int((right[face - 1] > 0).sum())
    charge = 48 * len(left) + 16 * entries + 32 * len(left) + 16 * m.n_elems + 4 * len(t.array("sub_elem_vert"))
    before = m.device_bytes
    b = LagBatch(capacity=1, budget_bytes=before + charge + 8 * 14 * m.n_elems)
    sol = np.zeros((m.n_elems, 5))
    sol[:, 0], sol[:, 4] = 1.0, 2.5
    assert b.add(m, sol, 1.0, cfl=0.5) is not None
    assert m.device_bytes - before == charge
    b.close()
