"""Concurrent queries, plain and pruned, on one handle, whose scans are answered by the coordinator or, when
several are in flight, by the merge tree alone: every thread's results against the oracle,
bit for bit, over table sizes and k on both sides of that choice."""
import threading

import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [130_000, 1_050_003, 6_000_011])
@pytest.mark.parametrize("threads", [2, 3, 8])
def test_threads_on_one_handle(n, threads):
    d = 4
    rng = np.random.default_rng([n, threads])
    x = rng.random((d, n), dtype=np.float32)
    x[:, ::97] = np.floor(x[:, ::97] * 8) / np.float32(8)
    queries = []
    for k in (1, 32, 64, 65, 300, 511, 512):
        for q in (1, 2, 4):
            w = (1 - rng.random(d)).astype(np.float32)
            a = rng.permutation(d)[:q].astype(np.uint8)
            queries.append((k, w, a, O.topk_numpy(x, k, w, a)))
    errors = []
    with T.Table(n, d) as t:
        t.upload(x)
        t.build_partitions(1024, T.ORDER_KD)

        def work(i):
            try:
                for j in range(3 * len(queries)):
                    k, w, a, want = queries[(i + j) % len(queries)]
                    H.assert_same_result(t.query(k, w, a), want)
                    H.assert_same_result(t.query_pruned(k, w, a)[:3], want)
            except Exception as e:  # reported below
                errors.append(e)

        pool = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
        for p in pool:
            p.start()
        for p in pool:
            p.join()
    assert not errors, errors[0]
