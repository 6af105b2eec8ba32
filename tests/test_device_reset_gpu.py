"""Handles made after the program reset its CUDA context (cudaDeviceReset, which ends only the calling
process's own) work like the first ones: nothing of the library's that handles share is left behind in
the old context. In a process of its own."""
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import ctypes
import numpy as np
import casim_b200 as cb
from casim_b200 import configs

def run():
    p, s = configs.small_mixed(n_sites=2, dim=3, cytosol="RD3D")
    out = []
    for path in ("plain", "resident"):
        sim = cb.ReleaseSiteBatch(p, s, path=path)
        sim.start(s["first_channel"])
        sim.step(20)
        out.append(sim.field(0, 0))
        sim.close()
    h = ctypes.c_void_p()
    assert cb.lib().casim_b200_sg_create(8, 4, 64, 1, 1, ctypes.byref(h)) == cb.OK
    assert cb.lib().casim_b200_sg_check(h) == cb.OK
    cb.lib().casim_b200_sg_destroy(h)
    return out

a = run()
cudart = ctypes.CDLL("libcudart.so.12")
assert cudart.cudaDeviceReset() == 0
b = run()
assert all(np.array_equal(x, y) for x, y in zip(a, b))
print("same")
"""


def test_handles_after_a_context_reset(cuda_device):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
