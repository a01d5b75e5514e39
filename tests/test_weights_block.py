"""Simple-kriging weights on both sides of the one-block kernel's limit of 160
neighbours (and of the 48 kB of shared memory a launch gets without asking,
75 neighbours), with the bound of tests/test_sk_weights.py: the device
evaluates exp and pow, so a weight may differ in its last bits.  Up to 64
neighbours against the oracle; above, which the oracle does not take, against
numpy's solution of the same system in 64 bits."""

import math

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W
from oracle import oracle as O


def _numpy_weights(c, pts, ct):
    """Covariance models of W.cov_params(ct, (12, 9, 7), angles=(20, 10, 5),
    nugget=0.1), the rotation as cov_model.h:16-61 builds it."""
    a0, a1, a2 = (math.radians(v) for v in (20, 10, 5))
    rz = np.array([[math.cos(a0), math.sin(a0), 0], [-math.sin(a0), math.cos(a0), 0], [0, 0, 1]])
    ry = np.array([[math.cos(a1), 0, -math.sin(a1)], [0, 1, 0], [math.sin(a1), 0, math.cos(a1)]])
    rx = np.array([[1, 0, 0], [0, math.cos(a2), math.sin(a2)], [0, -math.sin(a2), math.cos(a2)]])
    t = np.diag([1.0, 12 / 9, 12 / 7]) @ (rx @ ry @ rz)

    def cov(d):
        h = np.sqrt(((d @ t.T) ** 2).sum(-1)) / 12
        v = np.where(h > 1, 0, 1 - 1.5 * h + 0.5 * h ** 3) if ct == 0 else np.exp(-3 * h ** ct)
        return 0.9 * v
    p = pts.astype(np.float64)
    return np.linalg.solve(cov(p[:, None] - p[None]), cov(p - c.astype(np.float64)))


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["hpgl_simple_kriging_weights", "hpgl_b200_simple_kriging_weights_static"])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 32, 33, 64, 75, 76, 159, 160, 161])
def test_weights_at_the_block_kernels_edges(native_lib, n, entry):
    rng = np.random.default_rng(n)
    side = 10.0 * n ** (1.0 / 3.0)
    pts = rng.uniform(0, side, (n, 3)).astype(np.float32)
    c = rng.uniform(0, side, 3).astype(np.float32)
    for ct in (0, 1, 2):
        p = W.cov_params(ct, (12, 9, 7), angles=(20, 10, 5), nugget=0.1)
        if n <= 64:
            rc, wo = O.sk_weights(c, pts[:, 0], pts[:, 1], pts[:, 2], p)
            assert rc == 0
        else:
            wo = _numpy_weights(c, pts, ct)
        wg = N.sk_weights(c, pts[:, 0], pts[:, 1], pts[:, 2], p, entry=entry)
        assert np.max(np.abs(wg - wo)) <= 1e-6 * max(1e-3, float(np.max(np.abs(wo))))


@pytest.mark.gpu
def test_weights_of_a_singular_system(native_lib):
    """Two neighbours in one place: refused, and the next query is not."""
    p = W.cov_params(1, (12, 9, 7))
    x = np.array([1.0, 1.0, 5.0], dtype=np.float32)
    with pytest.raises(N.HpglError):
        N.sk_weights((0, 0, 0), x, x, x, p)
    assert np.isfinite(N.sk_weights((0, 0, 0), x[1:], x[1:], x[1:], p)).all()
