"""The clusterizer search's early drop of candidates beyond the model's reach:
the limit against the model on the host (tests/cpp/plan_reach_check.cpp), and
whole neighbour lists against the oracle on jobs whose every node takes the
clusterizer path with candidates on both sides of the limit."""

import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O
from tests.helpers import f32_bits_equal, neighbour_lists_equal

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_limit_keeps_what_the_filter_keeps(tmp_path):
    out = str(tmp_path / "plan_reach_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-o", out,
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "cpp", "plan_reach_check.cpp"),
                    os.path.join(ROOT, "hpgl_b200", "csrc", "plan.cpp"),
                    os.path.join(ROOT, "hpgl_b200", "csrc", "task_pool.cpp")], check=True, capture_output=True)
    kept, dropped = C.c_longlong(), C.c_longlong()
    assert C.CDLL(out).prc_run(17, 300, C.byref(kept), C.byref(dropped)) == 0
    assert kept.value > 100000 and dropped.value > 100000


def _model(cov, ranges, angles):
    """C(d) / C(0) of offsets d, the rotation as cov_model.h:16-61 builds it."""
    a0, a1, a2 = (math.radians(v) for v in angles)
    rz = np.array([[math.cos(a0), math.sin(a0), 0], [-math.sin(a0), math.cos(a0), 0], [0, 0, 1]])
    ry = np.array([[math.cos(a1), 0, -math.sin(a1)], [0, 1, 0], [math.sin(a1), 0, math.cos(a1)]])
    rx = np.array([[1, 0, 0], [0, math.cos(a2), math.sin(a2)], [0, -math.sin(a2), math.cos(a2)]])
    t = np.diag([1.0, ranges[0] / ranges[1], ranges[0] / ranges[2]]) @ (rx @ ry @ rz)

    def f(d):
        h = np.sqrt(((d @ t.T) ** 2).sum(-1)) / ranges[0]
        return np.where(h > 1, 0, 1 - 1.5 * h + 0.5 * h ** 3) if cov == 0 else np.exp(-3 * h ** cov)
    return f


SHAPE, RADII, ANGLES = (37, 33, 9), (8, 7, 4), (25, 10, 5)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ok", "sk"])
@pytest.mark.parametrize("cov", [0, 1, 2])
@pytest.mark.parametrize("ranges", [(9, 9, 9), (12, 6, 5), (6, 300, 4), (5000, 8, 6), (9, 5, 40)])
def test_lists_on_both_sides_of_the_limit(native_lib, kind, cov, ranges):
    model = _model(cov, ranges, ANGLES)
    grid = np.stack(np.meshgrid(*[np.arange(-r, r + 1) for r in RADII], indexing="ij"), -1).reshape(-1, 3)
    limit = int((model(grid) > 0.01).sum()) // 250  # informed nodes a box takes
    assert limit >= 1
    # up to two informed nodes a box: no box is too full, and the 54 of the 27
    # boxes all fit the list, so that a dropped one is missed
    rng = np.random.default_rng(cov)
    nx, ny, nz = SHAPE
    nodes = np.stack([np.arange(nx * ny * nz) % nx, np.arange(nx * ny * nz) // nx % ny,
                      np.arange(nx * ny * nz) // (nx * ny)], 1)
    box = nodes // np.array(RADII)
    mask = np.zeros(len(nodes), np.uint8)
    held = {}
    for i in rng.permutation(len(nodes)):
        b = tuple(box[i])
        if held.get(b, 0) < min(limit, 2):
            held[b] = held.get(b, 0) + 1
            mask[i] = 1
    points = np.nonzero(mask)[0]
    d = nodes[:, None] - nodes[points][None]
    near = (np.abs(box[:, None] - box[points][None]) <= 1).all(-1)
    c = model(d)
    # in terms of distance: a limit 10 % too near would cut the first, and the second must go
    assert (near & (c > 0.01) & (model(d / 0.9) <= 0.01)).sum() > 100
    assert (near & (c <= 0.01)).sum() > 100
    values = np.where(mask > 0, rng.standard_normal(len(nodes)), -99).astype(np.float32)
    p = W.cov_params(cov, ranges, angles=ANGLES, sill=1.0, nugget=0.1, radii=RADII, max_neighbours=64)
    job = dict(kind=kind, shape=SHAPE, mask=mask, values=values, params=[p], sk_mean=0.1)
    ref = O.run(job, kind=kind)
    got = N.krige(job, precision="fp64", kind=kind, dumps=True)
    sr = np.nonzero(ref["status"] >= 0)[0]
    assert not ref["via_template"][sr].any()
    assert np.array_equal(ref["status"], got["status"])
    ok, msg = neighbour_lists_equal(ref, got, sr, sr, ref["cap"], got["cap"])
    assert ok, msg
    assert f32_bits_equal(got["out"], ref["out"])
