"""A state may outlive its mesh, with steps still queued: its memory goes back to the pool
only after them, so that the next state's results are its own; also with mesh and state
closed from two threads."""
import threading

import numpy as np
import pytest

from test_ns_gpu import _perturbed_gresho

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [False, True])
def test_state_outlives_its_mesh(native, cuda_ok, threads):
    from subfv_b200 import meshgen
    from subfv_b200.mesh import Mesh
    from subfv_b200.ns import NsConfig, NsState
    cfg = NsConfig(scheme=1, second_order=True, method=4, bc_style=2, cfl=0.4)
    raw = meshgen.hex_slab(160, 150, jitter=0.1, seed=5)
    m = Mesh.from_raw(raw)
    sol = _perturbed_gresho(m, 3)

    def run():
        s = NsState(m, cfg, sol)
        out = s.advance(3), s.sol()
        s.close()
        return out

    ref = run()
    for _ in range(3):
        gone = Mesh.from_raw(raw)
        old = NsState(gone, cfg, sol)
        old.prepare()
        old.advance_async(200)
        if threads:
            both = [threading.Thread(target=x.close) for x in (gone, old)]
            for t in both:
                t.start()
            for t in both:
                t.join()
        else:
            gone.close()
            old.close()
        got = run()
        assert got[0] == ref[0]
        np.testing.assert_array_equal(got[1], ref[1])
