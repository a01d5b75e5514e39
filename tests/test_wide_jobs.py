"""Jobs whose neighbour offsets do not pack into one 32-bit word (OffsetPack):
the one-system-a-warp kernels solve them.  4097x65x65 with the untruncated model
over the whole grid is about the smallest: each field holds the largest
difference plus the range, 15 + 9 + 9 bits.  A sample of nodes against the
oracle, bit for bit."""

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O
from tests.helpers import f32_bits_equal

pytestmark = pytest.mark.gpu

SHAPE = (4097, 65, 65)


def _sample(mask, count):
    rng = np.random.default_rng(9)
    nodes = rng.choice(mask.size, 4 * count, replace=False)
    return np.sort(nodes[mask[nodes] == 0][:count]).astype(np.int32)


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
    assert got["top_kernel"] == "k_solve_exact32"
    nodes = _sample(mask, 1500)
    ref = O.run(job, kind="ok", dumps=False, node_list=nodes)
    assert np.array_equal(got["out_mask"][nodes], ref["out_mask"][nodes])
    assert f32_bits_equal(got["out"][nodes], ref["out"][nodes])


def test_wide_cokriging(native_lib):
    job = W.cokriging_job(shape=SHAPE, seed=2, informed=0.3, max_neighbours=8)
    # the template spans the grid: pairs of neighbours reach twice its extent
    job["params"] = [dict(job["params"][0], cov_type=1, ranges=(4000.0, 60.0, 60.0), radii=(2048, 32, 32))]
    _, got = N.bench(job, precision="fp64", iters=1, warmup=0)
    assert got["top_kernel"] == "k_cokriging"
    nodes = _sample(job["mask"], 1500)
    ref = O.cokriging(job, dumps=False, node_list=nodes)
    assert np.array_equal(got["out_mask"][nodes], ref["out_mask"][nodes])
    assert f32_bits_equal(got["out"][nodes], ref["out"][nodes])
