"""The device memory that variogram calls keep for the next one: bounded, and
given back on request.  In a process of its own, so that little else moves the
device's free memory: the driver's own pages for the process still do, 64 kB at
a time, while a pool takes and returns memory in units of UNIT bytes."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
UNIT = 2 << 20  # the granularity of device allocations (cuMemGetAllocationGranularity)

CHILD = """
import ctypes as C
import numpy as np
from hpgl_b200 import cvariogram as CV
cuda = C.CDLL("libcuda.so.1")
def free():
    f, t = C.c_size_t(), C.c_size_t()
    assert cuda.cuMemGetInfo_v2(C.byref(f), C.byref(t)) == 0
    return f.value
def call(shape):
    rng = np.random.default_rng(1)
    v = rng.standard_normal(shape).astype(np.float32)
    t = CV.VariogramSearchTemplate(5, 5, 0.3, 4, 0, CV.Ellipsoid(20, 4, 4, 30, 0, 0))
    return CV.CalcVariogramStats(t, hard_data=(v, np.ones(shape, np.uint8)))
CV.ReleaseMemory()
first = call((4, 4, 4))
CV.ReleaseMemory()
before = free()
big = call((60, 500, 400))
kept = before - free()
CV.ReleaseMemory()
after = before - free()
huge = call((60, 2000, 1200))
kept_huge = before - free()
CV.ReleaseMemory()
again = call((4, 4, 4))
assert all(np.array_equal(a, b) for a, b in zip(first, again))
CV.ReleaseMemory()
print(kept, after, kept_huge, before - free())
"""


@pytest.mark.gpu
def test_kept_memory(native_lib):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stderr
    kept, after, kept_huge, end = (int(x) for x in r.stdout.split())
    assert kept >= UNIT and after < UNIT and end < UNIT, r.stdout
    # 256 MB stay, and what the device rounds an allocation up to
    assert kept_huge <= (256 << 20) + (64 << 20), r.stdout
