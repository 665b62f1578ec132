"""A kernel that asks for more than 48 KB of shared memory needs the limit
raised in the context it is launched in: an engine made in a second context
(after the first was reset, or on a second device) has to run like the first.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

# 850,000 atoms on: the mixed force pass with its tables in shared memory
CHILD = """
import ctypes, sys
import numpy as np
from moldy_b200 import MoldySystem, workloads as wl
w = wl.make_workload(76, sigma=0.05, temperature=300.0, ivol=1, seed=3)

def evaluate(device):
    g = MoldySystem.from_workload(w, precision="mixed", device=device)
    pe = g.force()["pe"]
    f = g.forces()
    g.close()
    return pe, f

pe, f = evaluate(0)
second = int(sys.argv[1])
if second == 0:
    assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
pe2, f2 = evaluate(second)
assert pe2 == pe and np.array_equal(f, f2)
print("same on the second context")
"""


def _child(second):
    r = subprocess.run([sys.executable, "-c", CHILD, str(second)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "same on the second context" in r.stdout, r.stdout + r.stderr


def test_shared_memory_limit_after_a_context_reset(gpu_lib):
    _child(0)


def test_shared_memory_limit_on_a_second_device(gpu_lib):
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    _child(1)
