"""Variogram and stacking calls on pinned arrays: none of the library's copies
of a caller's array is still under way when the call returns, whichever way it
returns.  Shown by the device being idle then: waiting for it takes a small part
of what copying the array does."""

import time

import numpy as np
import pytest

import variogram_cases as VC
from tests.test_gpu_variogram import CV, gpu_template  # noqa: F401

pytestmark = pytest.mark.gpu

CELLS = 1 << 29  # bytes


@pytest.fixture(scope="module")
def pinned():
    import torch
    host = torch.zeros(CELLS, dtype=torch.uint8, pin_memory=True)
    dev = torch.empty(CELLS, dtype=torch.uint8, device="cuda")
    times = []
    for _ in range(3):
        torch.cuda.synchronize()
        t = time.perf_counter()
        dev.copy_(host, non_blocking=True)
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t)
    return host.numpy(), min(times)


def _wait():
    import torch
    t = time.perf_counter()
    torch.cuda.synchronize()
    return time.perf_counter() - t


# offsets of at least one cell along x, which a mask one cell wide pairs with nothing
BEYOND = (1.0, 1.0, 0.4, 3, 2.0, (6.0, 1.0, 1.0), (0.0, 0.0, 0.0))


def test_mask_narrower_than_every_offset(CV, pinned):  # noqa: F811
    host, copy = pinned
    sums, counts = CV.CalcVariogramStats(gpu_template(CV, BEYOND),
                                         hard_data=(np.ones((1, 1, 4), np.float32), host.reshape(1, 1, -1)))
    assert _wait() < 0.25 * copy
    assert not sums.any() and not counts.any()


def test_mask_smaller_than_the_data(CV, pinned):  # noqa: F811
    host, copy = pinned
    with pytest.raises(CV.HpglError):
        CV.CalcVariogramStats(gpu_template(CV, VC.TEMPLATES["x_narrow"]),
                              hard_data=(np.ones((2, 1, 4), np.float32), host.reshape(1, 1, -1)))
    assert _wait() < 0.25 * copy


def test_stack_deeper_than_the_result(CV, pinned):  # noqa: F811
    host, copy = pinned
    result = host.view(np.float32).reshape(64, 64, -1)
    layer = np.ones((64, 64), np.float32)
    with pytest.raises(CV.HpglError):
        CV.CStackLayers([layer], [1], result.shape[2] + 1, 1.0, 0, result)
    assert _wait() < 0.25 * copy


def test_negative_strides_stay_refused(CV):  # noqa: F811
    v, m = VC.grid((1, 5, 4), 1.0, seed=1)
    with pytest.raises(CV.HpglError):
        CV.CalcVariogramStats(gpu_template(CV, BEYOND), hard_data=(v, m[:, ::-1]))
