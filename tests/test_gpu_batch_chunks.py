"""Batches at the edges of the chunk schedule (quadrupling up to 2^16 results and k = 1024,
doubling above): table sizes around its boundaries, against the oracle, bit for bit."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 8192, 8193, 4 * 8192, 4 * 8192 + 1, 16 * 8192 - 1, 16 * 8192 + 257])
@pytest.mark.parametrize("nq,k", [(1, 1), (3, 1024), (3, 1025), (65, 1008), (66, 1008), (130, 500)])
@pytest.mark.parametrize("d", [5, 17])
def test_chunk_schedule(n, nq, k, d):
    rng = np.random.default_rng([n, nq, d])
    x = rng.random((d, n), dtype=np.float32)
    ks = np.full(nq, k, np.uint64)
    qqs = rng.integers(1, d, nq, endpoint=True).astype(np.uint32)
    w = rng.uniform(-0.3, 1, (nq, d)).astype(np.float32)
    a = rng.permuted(np.tile(np.arange(d, dtype=np.uint8), (nq, 1)), axis=1)
    with T.Table(n, d) as t:
        t.upload(x)
        ids, sc, cnt, th = t.query_batch(ks, w, a, qqs)
    for j in {0, nq // 2, nq - 1}:
        c = int(cnt[j])
        H.assert_same_result((ids[j, :c], sc[j, :c], th[j]), O.topk_numpy(x, k, w[j], a[j, :qqs[j]]))
