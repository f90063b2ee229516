"""The tile node kernel at the edges of its tiles, bit for bit against the oracle: meshes
whose vertex counts leave part of a tile empty or need a single vertex more than one tile,
wheels of k triangles (2 k subfaces and k corners around the hub: the classes of 8, 16 and
32 subfaces and the counts next to them), boxes, periodic boxes, every boundary style."""
import numpy as np
import pytest

from test_ns_gpu import _pair, _perturbed_gresho

pytestmark = pytest.mark.gpu


def wheel(k):
    """k prisms around a hub edge (a fan of k triangles on the unit circle, one layer)."""
    from subfv_b200 import meshgen
    a = 2 * np.pi * np.arange(k) / k
    xy = np.concatenate([[[0.03, 0.02]], 0.5 * np.column_stack([np.cos(a), np.sin(a)])])
    n = k + 1
    coords = np.column_stack([np.tile(xy, (2, 1)), np.repeat([-0.5, 0.5], n)])
    tri = np.column_stack([np.zeros(k, int), 1 + np.arange(k), 1 + (np.arange(k) + 1) % k])
    ev = np.concatenate([tri, tri + n], axis=1) + 1
    return meshgen.RawMesh(coords, np.full(k, meshgen.KIND_PRISM, np.int32), (np.arange(k + 1) * 6).astype(np.int32),
                           ev.astype(np.int32).ravel(), b2d=True)


def _raw(name):
    from subfv_b200 import meshgen
    kind, *n = name.split("_")
    n = [int(v) for v in n]
    if kind == "quads":
        return meshgen.hex_slab(*n, jitter=0.1, seed=3)
    if kind == "tris":
        return meshgen.prism_slab(*n, -0.5, 0.5, -0.5, 0.5, -0.5, 0.5, jitter=0.05, seed=4)
    if kind == "wheel":
        return wheel(*n)
    return meshgen.hex_box(n[0], jitter=0.05, seed=5, periodic=kind == "pbox")


@pytest.mark.parametrize("cfg", [dict(scheme=1, second_order=True, bc_style=2), dict(scheme=1, second_order=False, bc_style=1),
                                 dict(scheme=1, second_order=False, bc_style=0), dict(scheme=4, second_order=True, bc_style=2)],
                         ids=["mp_o2_bc2", "mp_o1_bc1", "mp_o1_bc0", "tw_o2"])
@pytest.mark.parametrize("name", ["quads_1_1", "quads_3_1", "quads_15_3", "quads_31_1", "tris_1_1", "tris_7_5", "tris_31_2",
                                  "wheel_3", "wheel_4", "wheel_5", "wheel_8", "wheel_9", "wheel_16", "box_2", "box_5",
                                  "pbox_4"])
def test_tile_edges_bit_exact(native, oracle_lib, cuda_ok, name, cfg):
    from subfv_b200.ns import NsConfig, compute_rhs_ns
    m, o = _pair(_raw(name))
    c = NsConfig(**cfg, method=4, boundary_2d="box" not in name, cfl=0.4)
    sol = _perturbed_gresho(m, 6)
    st, rhs, sl, vp, grad = compute_rhs_ns(m, c, sol)
    st_o, rhs_o, sl_o, vp_o, grad_o = o.ns_rhs(c.oracle_dict(), sol)
    assert st == st_o
    np.testing.assert_array_equal(sl, sl_o)
    np.testing.assert_array_equal(rhs, rhs_o)
    if c.scheme == 1:
        np.testing.assert_array_equal(vp, vp_o)
