"""The clusterizer search's ordering (k_search_cluster): whole neighbour lists
against the oracle, which sorts with std::sort, on isotropic models whose
symmetric offsets tie, at the sizes where the ordering changes its ways: parts
of 16, partitions of 64, lists shorter and longer than the candidates."""

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O
from tests.helpers import f32_bits_equal, neighbour_lists_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [1, 15, 16, 17, 18, 32, 33, 63, 64, 65, 66, 80, 81, 130, 400])
@pytest.mark.parametrize("nmax", [1, 16, 48, 49, 64])
def test_lists_match_std_sort(native_lib, points, nmax):
    rng = np.random.default_rng(100 * points + nmax)
    shape = (15, 14, 9)
    size = int(np.prod(shape))
    mask = np.zeros(size, np.uint8)
    mask[rng.choice(size, points, replace=False)] = 1
    values = np.where(mask > 0, rng.standard_normal(size), -99).astype(np.float32)
    # ranges far beyond the grid keep every candidate; the radii make a
    # template of over 100 000 entries, so that no box is too full
    p = W.cov_params(1, (40, 40, 40), sill=1.0, nugget=0.1, radii=(31, 31, 31), max_neighbours=nmax)
    job = dict(kind="ok", shape=shape, mask=mask, values=values, params=[p])
    ref = O.run(job, kind="ok")
    got = N.krige(job, precision="fp64", kind="ok", dumps=True)
    sr = np.nonzero(ref["status"] >= 0)[0]
    assert np.array_equal(ref["status"], got["status"])
    ok, msg = neighbour_lists_equal(ref, got, sr, sr, ref["cap"], got["cap"])
    assert ok, msg
    assert f32_bits_equal(got["out"], ref["out"])


@pytest.mark.parametrize("kind", ["ok", "sk"])
@pytest.mark.parametrize("cov", [0, 1, 2])
@pytest.mark.parametrize("ranges", [(9, 9, 9), (12, 5, 3), (3, 200, 1), (0.004, 5, 5), (5000, 2, 2)])
def test_candidates_within_reach(native_lib, kind, cov, ranges):
    # the candidates that are dropped before their covariance is read are
    # those it would drop, at skewed and extreme anisotropies
    rng = np.random.default_rng(cov)
    shape = (37, 33, 9)
    size = int(np.prod(shape))
    mask = (rng.random(size) < 0.02).astype(np.uint8)
    values = np.where(mask > 0, rng.standard_normal(size), -99).astype(np.float32)
    p = W.cov_params(cov, ranges, angles=(25, 10, 5), sill=1.0, nugget=0.1, radii=(30, 31, 32), max_neighbours=20)
    job = dict(kind=kind, shape=shape, mask=mask, values=values, params=[p], sk_mean=0.1)
    ref = O.run(job, kind=kind)
    got = N.krige(job, precision="fp64", kind=kind, dumps=True)
    sr = np.nonzero(ref["status"] >= 0)[0]
    assert np.array_equal(ref["status"], got["status"])
    ok, msg = neighbour_lists_equal(ref, got, sr, sr, ref["cap"], got["cap"])
    assert ok, msg
    assert f32_bits_equal(got["out"], ref["out"])
