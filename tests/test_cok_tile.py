"""Cokriging on lane tiles (hpgl_b200/csrc/cok_tile.cuh) at the edges of every
tile size against the oracle, bit for bit, and the systems it leaves to the
one-system-a-warp kernel: vanishing pivots, pivots beyond its range, more than
48 neighbours.  Layout and reciprocals: tests/test_tile_solve.py."""

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O
from tests.test_gpu_cokriging import _compare

SIZES = [1, 2, 7, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 32, 33, 36, 37, 40, 41, 44, 45, 48, 49]


def _check(job):
    _compare(O.cokriging(job), N.krige(job, dumps=True))


@pytest.mark.gpu
@pytest.mark.parametrize("mark", [1, 2])
@pytest.mark.parametrize("nmax", SIZES)
def test_cok_tile_edges(native_lib, nmax, mark):
    _check(W.cokriging_job(shape=(19, 13, 7), mark=mark, seed=nmax, informed=0.15, max_neighbours=nmax))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,informed", [((3, 2, 1), 0.3), ((33, 5, 2), 0.01), ((11, 7, 3), 0.95)])
def test_cok_tile_ragged_jobs(native_lib, shape, informed):
    for nmax in (8, 24, 48):
        _check(W.cokriging_job(shape=shape, seed=4, informed=informed, max_neighbours=nmax))


@pytest.mark.gpu
@pytest.mark.parametrize("nmax", [8, 20, 36])
def test_cok_tile_vanishing_pivots(native_lib, nmax):
    """Covariances all equal to C(0): every system with two neighbours or more
    loses a pivot."""
    job = W.cokriging_job(shape=(14, 12, 5), seed=9, informed=0.1, max_neighbours=nmax)
    job["params"] = [dict(job["params"][0], cov_type=2, ranges=(1e9, 1e9, 1e9))]
    _check(job)


@pytest.mark.gpu
@pytest.mark.parametrize("sill", [1e-280, 1e280])
def test_cok_tile_pivots_beyond_its_range(native_lib, sill):
    job = W.cokriging_job(shape=(14, 12, 5), seed=10, informed=0.1, max_neighbours=16)
    job["params"] = [dict(job["params"][0], sill=sill)]
    _check(job)
