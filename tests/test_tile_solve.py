"""The tiled solves (hpgl_b200/csrc/tile_solve.cuh): their shared-memory
layout and packed offsets on the host, their pivot arithmetic against CUDA's
IEEE operations, and whole jobs at the edges of every tile size against the
oracle, bit for bit."""

import os
import subprocess
import tempfile

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O
from tests.helpers import f32_bits_equal, neighbour_lists_equal

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tile_layout_and_packed_offsets():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "tile_geom_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "tile_geom_check.cpp")],
                       check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_pivot_root_and_reciprocal_match_ieee():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "pivot_check")
        subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3",
                        "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "pivot_check.cu")], check=True)
        r = subprocess.run([exe, "100000000"], capture_output=True, text=True, timeout=300)
        print(r.stdout)
        assert r.returncode == 0, r.stdout + r.stderr


def _job(kind, nmax, shape, informed, seed, cov=1, sill=1.0):
    rng = np.random.default_rng(seed)
    size = int(np.prod(shape))
    mask = (rng.random(size) < informed).astype(np.uint8)
    p = W.cov_params(cov, (6, 5, 4), angles=(25, 0, 0), sill=sill, nugget=0.02 * sill, radii=(7, 6, 5),
                     max_neighbours=nmax, marginal_prob=0.4)
    job = dict(kind=kind, shape=shape, mask=mask, params=[p], sk_mean=0.25)
    if kind in ("ik", "median_ik"):
        job["codes"] = rng.integers(0, 2, size).astype(np.uint8)
        job["params"] = [p, dict(p, marginal_prob=0.6)] if kind == "ik" else [p]
    else:
        job["values"] = np.where(mask > 0, rng.standard_normal(size), -99).astype(np.float32)
        job["mean"] = rng.normal(0, 0.3, size).astype(np.float32)
    return job


def _check(job, kind):
    ref = O.run(job, kind=kind)
    got = N.krige(job, precision="fp64", kind=kind, dumps=True)
    nodes = np.arange(int(np.prod(job["shape"])))
    sr = nodes * 2 if kind == "ik" else np.nonzero(ref["status"] >= 0)[0]
    sg = nodes if kind == "ik" else sr
    assert np.array_equal(ref["out_mask"], got["out_mask"])
    assert np.array_equal(ref["status"][sr], got["status"][sg])
    ok, msg = neighbour_lists_equal(ref, got, sr, sg, ref["cap"], got["cap"])
    assert ok, msg
    assert np.array_equal(ref["out"], got["out"]) if kind in ("ik", "median_ik") else f32_bits_equal(ref["out"], got["out"])
    solved = ref["status"][sr] == 0
    assert np.array_equal(ref["variance"][sr][solved].view(np.uint64), got["variance"][sg][solved].view(np.uint64))
    cap = ref["cap"]
    valid = np.arange(cap)[None, :] < ref["nb_count"][sr][solved][:, None]
    rw = ref["weights"].reshape(-1, cap)[sr][solved]
    gw = got["weights"].reshape(-1, got["cap"])[sg][solved][:, :cap]
    assert np.array_equal(rw[valid].view(np.uint64), gw[valid].view(np.uint64))


SIZES = [1, 2, 7, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 31, 32]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ok", "sk", "lvm", "ik", "median_ik"])
@pytest.mark.parametrize("nmax", SIZES)
def test_tile_edges_match_the_oracle(native_lib, nmax, kind):
    """An odd grid, dense enough that most systems are full, with ragged
    counts at its faces."""
    _check(_job(kind, nmax, (19, 13, 9), 0.12, 100 + nmax), kind)


WIDE = [33, 36, 37, 40, 41, 44, 45, 48, 49, 52, 53, 56, 57, 63, 64]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["ok", "sk", "ik"])
@pytest.mark.parametrize("nmax", WIDE)
def test_wide_tile_edges_match_the_oracle(native_lib, nmax, kind):
    _check(_job(kind, nmax, (15, 11, 7), 0.2, 200 + nmax), kind)


@pytest.mark.gpu
@pytest.mark.parametrize("nmax", [40, 48, 64])
def test_wide_singular_systems_keep_their_status(native_lib, nmax):
    job = _job("ok", nmax, (16, 12, 8), 0.2, 6, cov=2)
    job["params"] = [dict(job["params"][0], ranges=(90.0, 90.0, 30.0), nugget=0.0)]
    _check(job, "ok")


@pytest.mark.gpu
@pytest.mark.parametrize("shape,informed", [((1, 1, 1), 1.0), ((3, 1, 1), 0.5), ((5, 2, 1), 0.3), ((33, 1, 2), 0.05),
                                            ((17, 11, 5), 0.002), ((11, 7, 3), 0.95)])
def test_tile_ragged_and_tiny_jobs(native_lib, shape, informed):
    """Fewer nodes than a warp has systems, systems with no neighbour, warps
    with idle groups."""
    for nmax in (8, 20, 32):
        for kind in ("ok", "sk"):
            _check(_job(kind, nmax, shape, informed, 7), kind)


@pytest.mark.gpu
@pytest.mark.parametrize("sill", [1e-200, 1e-30, 1e30, 1e220])
def test_sills_at_the_ends_of_the_range(native_lib, sill):
    """Pivots far from 1, and beyond the range of the tiled kernels' pivot
    arithmetic (the one-system-a-warp kernel takes those jobs)."""
    _check(_job("sk", 20, (15, 12, 6), 0.1, 3, sill=sill), "sk")


@pytest.mark.gpu
@pytest.mark.parametrize("nmax", [12, 24, 32])
def test_singular_systems_keep_their_status(native_lib, nmax):
    """A long Gaussian model: some factorisations fail, others next to them in
    the same warp do not."""
    job = _job("ok", nmax, (16, 16, 8), 0.1, 5, cov=2)
    job["params"] = [dict(job["params"][0], ranges=(90.0, 90.0, 30.0), nugget=0.0)]
    _check(job, "ok")
