"""GPU test: a program that resets its device between two uses of the package
(cudaDeviceReset, which ends the process's own context) gets the same results
from handles made after it. In a process of its own: the reset takes every
allocation of the process with it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, glob, os, sys
import numpy as np
import stratiflow_b200 as sf

def run(cls):
    if cls == "ensemble":
        e = sf.Ensemble([(64, 64), (128, 128)], (14.0, 10.0, 1000.0, 1.0), 0.01)
        e.step(2)
        e.synchronize()
        x = [m.get_state_kept() for m in e.members]
        e.close()
        return x
    s = sf.IMEXRK(128, cls, 96, 14.0, 7.0, 10.0, 1000.0, 1.0, 0.01)
    rng = np.random.default_rng(1)
    x = (rng.standard_normal(s.kept_shape) * 1e-3).astype(np.complex64)
    s.set_state_kept(x)
    s.TimeStep(2)
    s.synchronize()
    x = s.get_state_kept()
    s.close()
    return [x]

kinds = (1, 16, "ensemble")
before = [run(k) for k in kinds]
import nvidia.cuda_runtime
rt = ctypes.CDLL(os.path.join(list(nvidia.cuda_runtime.__path__)[0], "lib", "libcudart.so.12"))
assert rt.cudaDeviceReset() == 0
after = [run(k) for k in kinds]
assert all(np.array_equal(a, b) for x, y in zip(before, after) for a, b in zip(x, y))
print("same")
"""


def test_handles_made_after_a_device_reset_work():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
