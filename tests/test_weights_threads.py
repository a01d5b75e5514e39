"""The two weights entries called at the same time: each is serialised with
itself only, so the block kernel they share must not take a setting of one call
into the other's launch.  Counts on both sides of the 48 kB of shared memory
that a launch gets without asking."""

import threading

import numpy as np
import pytest

from hpgl_b200 import native as N
from hpgl_b200 import workloads as W


def _query(n):
    rng = np.random.default_rng(n)
    pts = rng.uniform(0, 10.0 * n ** (1.0 / 3.0), (n, 3)).astype(np.float32)
    return pts[0] + np.float32(0.5), pts[:, 0].copy(), pts[:, 1].copy(), pts[:, 2].copy(), \
        W.cov_params(1, (12, 9, 7), angles=(20, 10, 5), nugget=0.1)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(160, 80), (80, 160), (160, 24)])
def test_both_entries_at_once(native_lib, sizes):
    entries = ("hpgl_simple_kriging_weights", "hpgl_b200_simple_kriging_weights_static")
    queries = [_query(n) for n in sizes]
    alone = [N.sk_weights(*q, entry=e) for q, e in zip(queries, entries)]
    errors = []
    start = threading.Barrier(2)

    def calls(k):
        start.wait()
        for _ in range(2000):
            try:
                w = N.sk_weights(*queries[k], entry=entries[k])
            except N.HpglError as e:
                errors.append((entries[k], str(e)))
                return
            if not np.array_equal(w.view(np.uint32), alone[k].view(np.uint32)):
                errors.append((entries[k], "weights differ"))
                return

    threads = [threading.Thread(target=calls, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
