"""The device memory of a simulation's scratch, which is kept between calls:
neighbour lists by window slot are taken where a kernel reads them (the lane
tiles) and for as many slots as there are nodes to simulate.  Each case in a
process of its own, as the scratch only grows."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes as C, sys
from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from tests.sis_cases import BASE, case, means
cuda = C.CDLL("libcuda.so.1")
def free():
    f, t = C.c_size_t(), C.c_size_t()
    assert cuda.cuMemGetInfo_v2(C.byref(f), C.byref(t)) == 0
    return f.value
def run():
    if sys.argv[1] == "correlogram":
        c = case(shape=(18, 16, 6), K=3, seed=5)
        ps = [dict(BASE, max_neighbours=12, marginal_prob=0.3) for _ in range(3)]
        N.simulate_indicator(dict(c, params=ps), 5, category_means=means(c["shape"], 3), correlogram=True)
    else:
        j = W.ok_50x50x20(shape=(18, 16, 6), seed=4)
        j["params"] = [dict(j["params"][0], max_neighbours=int(sys.argv[1]), radii=(6, 6, 4))]
        N.simulate(j, 7, kind="sk")
L = N.lib()
run()
before = free()
L.hpgl_b200_set_sim_window(int(sys.argv[2]))
run()
print("grown", before - free())
"""


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["40", "32", "correlogram"])
def test_scratch_of_a_wide_window(native_lib, case):
    # a slot costs 21 bytes without its list, and a list 4 bytes a neighbour
    window = 1 << 23
    r = subprocess.run([sys.executable, "-c", CHILD, case, str(window)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split()[-1]) < 32 * window, r.stdout
