"""Batches over a table whose later rows score higher: queries stay on the tensor-core filter
as long as a chunk of twice the rows seen would not hold 2k + 2048 of their candidates."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [100, 372, 373, 1024])
def test_rising_scores_stay_on_the_filter(k):
    n, d, nq = 8192 * 20, 4, 40
    rng = np.random.default_rng(k)
    x = rng.random((d, n), dtype=np.float32) * np.float32(0.01)  # the other columns: little noise
    u = rng.random(n, dtype=np.float32)
    # after the first 8192 rows 1.6 times as many rows above any high score
    x[0] = np.where(np.arange(n) < 8192, u, 1 - (1 - u) / np.float32(1.6))
    w = np.ones((nq, d), np.float32)
    a = np.tile(np.arange(d, dtype=np.uint8), (nq, 1))
    qqs = np.full(nq, d, np.uint32)
    with T.Table(n, d) as t:
        t.upload(x)
        ids, sc, cnt, th = t.query_batch(np.full(nq, k, np.uint64), w, a, qqs)
        st = t.last_batch_stats()
    assert st["method"] == T.BATCH_BF16 and st["switched_fp32"] == 0
    for j in (0, nq - 1):
        H.assert_same_result((ids[j], sc[j], th[j]), O.topk_numpy(x, k, w[j], a[j]))
