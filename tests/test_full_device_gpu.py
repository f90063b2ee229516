"""Coordinates can be read and set with no device memory left: the staging buffer they pass
through is a convenience. In a process of its own, which fills the device and ends."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
from subfv_b200 import meshgen
from subfv_b200.mesh import Mesh
raw = meshgen.prism_slab(300, 300, jitter=0.05, seed=2)
m = Mesh.from_raw(raw)
rt = ctypes.CDLL("libcudart.so.12")
held, size = [], 1 << 36
while size >= 1 << 16:
    p = ctypes.c_void_p()
    if rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
        held.append(p)
    else:
        size >>= 1
rt.cudaGetLastError()
x = m.coords()
y = x.copy()
y[:, 0] += 0.25
m.set_coords(y)
z = m.coords()
for p in held:
    rt.cudaFree(p)
np.testing.assert_array_equal(z, y)
np.testing.assert_array_equal(m.coords(), y)  # with room again
print("held", len(held), "ok")
"""


def test_coords_without_device_memory(native, cuda_ok):
    root = str(Path(__file__).resolve().parent.parent)
    p = subprocess.run([sys.executable, "-c", SCRIPT.format(root=root)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "ok" in p.stdout, p.stdout + p.stderr
