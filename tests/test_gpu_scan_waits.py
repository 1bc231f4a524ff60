"""Scans whose bounded waits run out: with a limit of a poll or a few (topk_set_wait_limit) the
CTAs and the coordinator give up on each other at any point and the merge tree answers, or
the coordinator still does; the scratch serves the next query all the same.  Against the
oracle, bit for bit, several times on one handle."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 400_000, 3_000_017])
@pytest.mark.parametrize("kind", ["uniform", "ties", "rising"])
def test_waits_that_run_out(n, kind):
    d = 4
    rng = np.random.default_rng([n, len(kind)])
    x = rng.random((d, n), dtype=np.float32)
    if kind == "ties":
        x = np.floor(x * 40) / np.float32(64)
    elif kind == "rising":
        x += np.linspace(0, 4, n, dtype=np.float32)
    queries = []
    for q in (1, 2, 4):
        for k in (1, 40, 300, 2500):
            w = (1 - rng.random(d)).astype(np.float32)
            a = rng.permutation(d)[:q].astype(np.uint8)
            queries.append((k, w, a, O.topk_numpy(x, k, w, a)))
    with T.Table(n, d) as t:
        t.upload(x)
        t.build_partitions(1024, T.ORDER_KD)
        for limit in (1, 2, 30, 0, 1, 0):  # 0: the default again
            t.set_wait_limit(limit)
            for k, w, a, want in queries:
                for _ in range(2):
                    H.assert_same_result(t.query(k, w, a), want)
                    H.assert_same_result(t.query_pruned(k, w, a)[:3], want)
