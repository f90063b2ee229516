"""The node kernels that serve multi_point and two_wave where the tiles do not: vertices with
more corners than their tile holds (two layers of a fan of k prisms: 3 k subfaces and 2 k
cells around the middle hub; k = 5, 9 and 10 do not fit), excluded boundary vertices, and
batches with such a mesh among others."""
from dataclasses import replace

import numpy as np
import pytest

from test_node_tile_gpu import wheel
from test_ns_gpu import _pair, _perturbed_gresho

pytestmark = pytest.mark.gpu


def two_layers(k):
    from subfv_b200 import meshgen
    raw = wheel(k)
    n = k + 1
    xy = raw.coords[:n, :2]
    coords = np.column_stack([np.tile(xy, (3, 1)), np.repeat([-0.5, 0.02, 0.5], n)])
    low = np.asarray(raw.elem_vert).reshape(k, 6)
    ev = np.concatenate([low, low + n])
    return meshgen.RawMesh(coords, np.full(2 * k, meshgen.KIND_PRISM, np.int32), (np.arange(2 * k + 1) * 6).astype(np.int32),
                           ev.astype(np.int32).ravel(), b2d=False)


CFGS = {"mp_o2": dict(scheme=1, second_order=True, bc_style=2), "mp_o1_bc1": dict(scheme=1, second_order=False, bc_style=1),
        "tw_o2": dict(scheme=4, second_order=True, bc_style=2)}


@pytest.mark.parametrize("cfg", list(CFGS))
@pytest.mark.parametrize("k", [4, 5, 8, 9, 10])
def test_corners_beyond_a_tile_bit_exact(native, oracle_lib, cuda_ok, k, cfg):
    from subfv_b200.ns import NsConfig, compute_rhs_ns
    m, o = _pair(two_layers(k))
    c = NsConfig(**CFGS[cfg], method=4, boundary_2d=False, cfl=0.4)
    sol = _perturbed_gresho(m, 6)
    st, rhs, sl, vp, grad = compute_rhs_ns(m, c, sol)
    st_o, rhs_o, sl_o, vp_o, grad_o = o.ns_rhs(c.oracle_dict(), sol)
    assert st == st_o
    np.testing.assert_array_equal(sl, sl_o)
    np.testing.assert_array_equal(rhs, rhs_o)
    if c.scheme == 1:
        np.testing.assert_array_equal(vp, vp_o)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("cfg", list(CFGS))
def test_layouts_agree_beyond_a_tile(native, cuda_ok, cfg, precision):
    """A thread per vertex and a group of lanes per vertex: the same bits at each level."""
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsConfig, NsState
    m = Mesh.from_raw(two_layers(9))
    c = NsConfig(**CFGS[cfg], method=4, boundary_2d=False, cfl=0.4, precision=precision, tmax=1e30)
    out = []
    for lanes in (0, 1):
        s = NsState(m, c, _perturbed_gresho(m, 6))
        s.set_node_kernel(lanes)
        out.append((s.advance(11), s.sol()))
        s.close()
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("name", ["quads", "box"])
def test_excluded_boundary_vertices_bit_exact(native, oracle_lib, cuda_ok, name):
    from subfv_b200 import meshgen
    from subfv_b200.ns import NsConfig, compute_rhs_ns
    raw = meshgen.hex_slab(9, 7, jitter=0.1, seed=3) if name == "quads" else meshgen.hex_box(4, jitter=0.05, seed=5, periodic=False)
    m, o = _pair(raw)
    c = NsConfig(scheme=1, second_order=True, method=4, bc_style=2, boundary_2d=name == "quads", cfl=0.4,
                 exclude_bound_vert=True)
    sol = _perturbed_gresho(m, 6)
    st, rhs, sl, _, _ = compute_rhs_ns(m, c, sol)
    st_o, rhs_o, sl_o, _, _ = o.ns_rhs(c.oracle_dict(), sol)
    assert st == st_o
    np.testing.assert_array_equal(sl, sl_o)
    np.testing.assert_array_equal(rhs, rhs_o)


@pytest.mark.parametrize("lanes", [0, 1])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_tiles_agree_with_the_other_kernels(native, cuda_ok, precision, lanes):
    """A periodic box has no boundary vertices, so excluding them changes nothing but the
    kernel that serves."""
    from subfv_b200 import meshgen
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsConfig, NsState, init_fourier_flow
    m = Mesh.from_raw(meshgen.hex_box(5, jitter=0.05, seed=3, periodic=True))
    c = NsConfig(scheme=1, second_order=True, method=4, bc_style=2, boundary_2d=False, cfl=0.4, precision=precision,
                 tmax=1e30)
    out = []
    for excl in (False, True):
        s = NsState(m, replace(c, exclude_bound_vert=excl), init_fourier_flow(m, seed=4))
        s.set_node_kernel(lanes)
        out.append((s.advance(11), s.sol()))
        s.close()
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("cfg", ["mp_o2", "tw_o2"])
def test_batch_of_both_kinds(native, cuda_ok, cfg):
    """The mesh beyond the tiles joins a batch and leaves it again; each problem ends with its
    solo state."""
    from subfv_b200 import meshgen
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsBatch, NsConfig, NsState
    c = NsConfig(**CFGS[cfg], method=4, boundary_2d=False, cfl=0.4)
    raws = [meshgen.hex_box(4, jitter=0.05, seed=5, periodic=False), two_layers(9), two_layers(5), two_layers(4)]
    meshes = [Mesh.from_raw(r) for r in raws]
    sols = [_perturbed_gresho(m, 7) for m in meshes]
    b = NsBatch(c, capacity=8, budget_bytes=1 << 32)
    slots, steps = {}, dict.fromkeys(range(4), 0)
    got = {}
    for joins, leaves, n in (([0], [], 9), ([1, 2], [], 17), ([], [1, 2], 8), ([3], [], 11), ([], [0, 3], 0)):
        for i in joins:
            slots[i] = b.add(meshes[i], sols[i], 1e30)
            assert slots[i] is not None
        for i in leaves:
            b.sync()
            got[i] = (b.info(slots[i]), b.sol(slots[i], meshes[i].n_elems))
            b.remove(slots.pop(i))
        b.advance(n)
        for i in slots:
            steps[i] += n
    b.sync()
    b.close()
    for i, ((t, n, _, st), sol) in got.items():
        s = NsState(meshes[i], replace(c, tmax=1e30), sols[i])
        assert (st, n, t) == s.advance(steps[i])
        np.testing.assert_array_equal(sol, s.sol())


def test_step_loop_captured_once_for_either_kind(native, cuda_ok):
    """A mesh beyond the tiles joins and leaves, several times: the loop with the tiles and the
    one without are each captured once."""
    from subfv_b200 import _lib, meshgen
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsBatch, NsConfig
    c = NsConfig(**CFGS["mp_o2"], method=4, boundary_2d=False, cfl=0.4)
    m, beyond = (Mesh.from_raw(r) for r in (two_layers(8), two_layers(9)))
    b = NsBatch(c, capacity=4, budget_bytes=1 << 32)
    assert b.add(m, _perturbed_gresho(m, 7), 1e30) is not None
    for _ in range(3):
        b.advance(8)
        k = b.add(beyond, _perturbed_gresho(beyond, 7), 1e30)
        b.advance(8)
        b.remove(k)
    b.sync()
    assert _lib.load().subfv_probe_ns_captures(b._h) == 2
    b.close()
