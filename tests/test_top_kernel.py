"""hpgl_b200_bench names the kernel that solved the job: the lane tiles, or the
one-system-a-warp kernels for the jobs the tiles do not take; and counts the
launches of a pass."""

import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W


@pytest.mark.gpu
@pytest.mark.parametrize("nmax, sill, kernel", [(12, 1.0, "k_solve_tile"), (40, 1.0, "k_solve_tile"),
                                                (12, 1e-250, "k_solve_exact32"), (40, 1e-250, "k_solve_exact64")])
def test_name_of_the_solve(native_lib, nmax, sill, kernel):
    job = W.ok_50x50x20(shape=(30, 28, 8))
    job["params"] = [dict(job["params"][0], max_neighbours=nmax, sill=sill)]
    assert N.bench(job, precision="fp64", iters=1, warmup=1)[1]["top_kernel"] == kernel


@pytest.mark.gpu
@pytest.mark.parametrize("nmax, kernel, launches", [(24, "k_cok_tile", 4), (49, "k_cokriging", 3)])
def test_launches_of_cokriging(native_lib, nmax, kernel, launches):
    # bit rows, search, elimination; after the tiles the nodes they marked
    job = W.cokriging_job(shape=(30, 28, 8), max_neighbours=nmax)
    info = N.bench(job, precision="fp64", iters=1, warmup=1)[1]
    assert (info["top_kernel"], info["launches"]) == (kernel, launches)
