"""The weights entries after the process has reset the device: both work in the
context that replaces the old one.  In a process of its own, as a reset ends
everything else that process holds on the device."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes as C, sys
import numpy as np
from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
cuda = C.CDLL("libcuda.so.1")
entries = ("hpgl_simple_kriging_weights", "hpgl_b200_simple_kriging_weights_static")
p = W.cov_params(1, (12, 9, 7), angles=(20, 10, 5), nugget=0.1)
def calls():
    out = []
    for n in (24, 160, 200):
        rng = np.random.default_rng(n)
        q = rng.uniform(0, 60, (n, 3)).astype(np.float32)
        out += [N.sk_weights((30, 30, 30), q[:, 0], q[:, 1], q[:, 2], p, entry=e) for e in entries]
    return out
first = calls()
for _ in range(2):
    assert cuda.cuDevicePrimaryCtxReset_v2(0) == 0
    again = calls()
    assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(first, again))
print("same")
"""


@pytest.mark.gpu
def test_entries_after_a_device_reset(native_lib):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
