"""Jobs on wide grids, whose neighbour offsets need more than 32 bits for the
range test of all three axes (OffsetPack): which pack all the same, on the host,
and a sample of nodes of two of them against the oracle, bit for bit.  4097x65x65
with the untruncated model over the whole grid is about the smallest: fields for
every difference and the range would need 15 + 9 + 9 bits."""

import os
import subprocess

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O
from tests.helpers import f32_bits_equal

HERE = os.path.dirname(os.path.abspath(__file__))
SHAPE = (4097, 65, 65)


def _sample(mask, count):
    rng = np.random.default_rng(9)
    nodes = rng.choice(mask.size, 4 * count, replace=False)
    return np.sort(nodes[mask[nodes] == 0][:count]).astype(np.int32)


def test_which_offsets_pack(tmp_path):
    exe = str(tmp_path / "offset_pack_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "offset_pack_check.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_wide_ordinary_kriging(native_lib):
    rng = np.random.default_rng(1)
    size = int(np.prod(SHAPE))
    mask = np.zeros(size, np.uint8)
    mask[rng.choice(size, 1500, replace=False)] = 1
    values = np.where(mask > 0, rng.standard_normal(size), -99).astype(np.float32)
    # few informed cells and a template of 100 000 entries: the clusterizer
    # path, whose pairs of neighbours reach 4 r - 2
    job = dict(kind="ok", shape=SHAPE, mask=mask, values=values,
               params=[W.cov_params(0, (300, 12, 12), radii=(1025, 17, 17), max_neighbours=8)])
    _, got = N.bench(job, precision="fp64", kind="ok", iters=1, warmup=0)
    assert got["top_kernel"] == "k_solve_tile"
    nodes = _sample(mask, 1500)
    ref = O.run(job, kind="ok", dumps=False, node_list=nodes)
    assert np.array_equal(got["out_mask"][nodes], ref["out_mask"][nodes])
    assert f32_bits_equal(got["out"][nodes], ref["out"][nodes])


@pytest.mark.gpu
def test_wide_cokriging(native_lib):
    job = W.cokriging_job(shape=SHAPE, seed=2, informed=0.3, max_neighbours=8)
    # the template spans the grid: pairs of neighbours reach twice its extent
    job["params"] = [dict(job["params"][0], cov_type=1, ranges=(4000.0, 60.0, 60.0), radii=(2048, 32, 32))]
    _, got = N.bench(job, precision="fp64", iters=1, warmup=0)
    assert got["top_kernel"] == "k_cok_tile"
    nodes = _sample(job["mask"], 1500)
    ref = O.cokriging(job, dumps=False, node_list=nodes)
    assert np.array_equal(got["out_mask"][nodes], ref["out_mask"][nodes])
    assert f32_bits_equal(got["out"][nodes], ref["out"][nodes])
