"""Grid variograms at the edges of the 32-cell words the pairs are found in:
rows around a multiple of 32 cells, a mask larger than the data, offsets longer
than the grid, empty and full masks.  Counts and exact sums as
tests/test_gpu_variogram.py."""

import numpy as np
import pytest

from oracle import oracle as O
import variogram_cases as VC
from tests.test_gpu_variogram import CV, gpu_template  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (5, 4, 3), (31, 6, 2), (32, 6, 2), (33, 6, 2), (63, 3, 3), (64, 3, 3), (65, 3, 3), (97, 2, 5)]


def _check(CV, spec, v, m, percent=100):  # noqa: F811
    o = O.variograms(O.cv_template(*spec), v, m, percent=percent)
    sums, counts = CV.CalcVariogramStats(gpu_template(CV, spec), hard_data=(v, m), percent=percent)
    assert np.array_equal(counts, o["counts"])
    assert np.array_equal(sums, o["exact_sums"])


@pytest.mark.parametrize("informed", [0.05, 0.4, 1.0])
@pytest.mark.parametrize("shape", SHAPES)
def test_word_edges(CV, shape, informed):  # noqa: F811
    for name in ("x_narrow", "overlapping_lags", "dipping"):
        v, m = VC.grid(shape, informed, seed=shape[0])
        _check(CV, VC.TEMPLATES[name], v, m)


def test_offsets_longer_than_the_grid(CV):  # noqa: F811
    spec = (8.0, 8.0, 0.8, 12, 0.0, (100.0, 9.0, 2.0), (-20.0, 0.0, 0.0))
    for shape in ((20, 7, 3), (40, 40, 2)):
        v, m = VC.grid(shape, 0.5, seed=3)
        _check(CV, spec, v, m)
        _check(CV, spec, v, m, percent=40)


def test_empty_mask(CV):  # noqa: F811
    v, m = VC.grid((40, 6, 2), 0.0, seed=4)
    sums, counts = CV.CalcVariogramStats(gpu_template(CV, VC.TEMPLATES["x_narrow"]), hard_data=(v, m))
    assert not sums.any() and not counts.any()


@pytest.mark.parametrize("outside", [0, 1])
def test_mask_larger_than_the_data(CV, outside):  # noqa: F811
    """The mask's cells outside the data's shape do not count, informed or not."""
    for shape, wider in (((31, 6, 3), (40, 6, 3)), ((33, 5, 4), (70, 9, 6)), ((64, 4, 2), (64, 5, 2))):
        v, m = VC.grid(shape, 0.6, seed=shape[0])
        big = np.full(wider, outside, np.uint8, order="F")
        big[tuple(slice(n) for n in shape)] = m
        for name in ("x_narrow", "overlapping_lags", "dipping"):
            for percent in (100, 40):
                t = gpu_template(CV, VC.TEMPLATES[name])
                got = CV.CalcVariogramStats(t, hard_data=(v, big), percent=percent)
                if percent == 100:
                    o = O.variograms(O.cv_template(*VC.TEMPLATES[name]), v, m)
                    assert np.array_equal(got[1], o["counts"]) and np.array_equal(got[0], o["exact_sums"])
                else:
                    # the sample is drawn by the mask's cell index
                    big0 = big.copy("F")
                    big0[shape[0]:] = 0
                    big0[:, shape[1]:] = 0
                    big0[:, :, shape[2]:] = 0
                    want = CV.CalcVariogramStats(t, hard_data=(v, big0), percent=percent)
                    assert np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])
