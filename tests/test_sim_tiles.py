"""Sequential simulation with its systems on lane tiles (k_sgs_search /
k_sgs_solve, k_sis_search / k_sis_solve / k_sis_draw), at the edges of every
tile size against the restatement: Gaussian values bit for bit, indicator codes
exactly, categories that share one search and system and categories that do
not, small windows, and a sill outside the tiled kernels' range."""

import numpy as np
import pytest

from hpgl_b200 import native as N
from oracle import oracle as O
from sis_cases import BASE, case, means
from tests.test_gpu_sgs import _job, _same

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 12, 13, 16, 17, 24, 25, 32]


@pytest.mark.parametrize("kind", ["sk", "ok"])
@pytest.mark.parametrize("nmax", SIZES)
def test_sgs_tile_edges(native_lib, nmax, kind):
    job = _job((21, 17, 7), seed=40 + nmax, n=nmax, radii=(9, 9, 4))
    r = N.simulate(job, 500 + nmax, kind=kind)
    v, m, _ = O.sgs(job, ordinary=kind == "ok", seed=500 + nmax)
    assert _same(r["out"], v) and np.array_equal(r["out_mask"], m)


@pytest.mark.parametrize("sill", [1e-250, 1.0])
def test_sgs_sill_range(native_lib, sill):
    job = _job((16, 14, 5), seed=3, n=20)
    job["params"] = [dict(job["params"][0], sill=sill)]
    r = N.simulate(job, 11, kind="sk")
    v, m, _ = O.sgs(job, seed=11)
    assert _same(r["out"], v) and np.array_equal(r["out_mask"], m)


@pytest.mark.parametrize("K", [2, 3, 5])
@pytest.mark.parametrize("nmax", [8, 12, 17, 32])
def test_sis_one_group(native_lib, nmax, K):
    """Categories with one covariance model and search: one system for all."""
    c = case(shape=(21, 17, 7), K=K, seed=nmax + K)
    ps = [dict(BASE, max_neighbours=nmax, marginal_prob=1.0 / K) for _ in range(K)]
    r = N.simulate_indicator(dict(c, params=ps), 91)
    codes, mask = O.sis(c["shape"], c["codes"], c["mask"], ps, seed=91)
    assert np.array_equal(r["out"], codes) and np.array_equal(r["out_mask"], mask)


@pytest.mark.parametrize("nmax", SIZES)
def test_sis_groups_apart(native_lib, nmax):
    c = case(shape=(19, 15, 6), K=3, seed=60 + nmax)
    ps = [dict(BASE, max_neighbours=nmax, marginal_prob=0.3), dict(BASE, max_neighbours=9, cov_type=1, marginal_prob=0.5),
          dict(BASE, max_neighbours=nmax, ranges=(5.0, 6.0, 3.0), marginal_prob=0.2)]
    r = N.simulate_indicator(dict(c, params=ps), 17)
    codes, mask = O.sis(c["shape"], c["codes"], c["mask"], ps, seed=17)
    assert np.array_equal(r["out"], codes) and np.array_equal(r["out_mask"], mask)


def test_sis_one_group_with_mean_cubes(native_lib):
    c = case(shape=(20, 16, 7), K=3, seed=71)
    ps = [dict(BASE, marginal_prob=0.0) for _ in range(3)]
    lv = means(c["shape"], 3)
    r = N.simulate_indicator(dict(c, params=ps), 5, category_means=lv, correlogram=False)
    codes, mask = O.sis(c["shape"], c["codes"], c["mask"], ps, seed=5, lvm=lv, correlogram=False)
    assert np.array_equal(r["out"], codes) and np.array_equal(r["out_mask"], mask)
