"""Batches when the memory for the tensor-core filter's records cannot be had (the failure
is made on the host): a table of 17 to 64 attributes is served by the FP32 scorer, and by
the filter again once memory is there; a table of up to 16 attributes reports it.  Results
against the oracle, bit for bit."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

TOPK_ERR_OOM = 3


def _batch(d, nq, rng):
    ks = rng.integers(1, 200, nq).astype(np.uint64)
    qqs = rng.integers(1, min(d, 32), nq, endpoint=True).astype(np.uint32)  # more run as single scans
    w = rng.uniform(-1, 1, (nq, d)).astype(np.float32)
    a = rng.permuted(np.tile(np.arange(d, dtype=np.uint8), (nq, 1)), axis=1)
    return ks, w, a, qqs


@pytest.mark.parametrize("d", [16, 17, 40])
def test_batch_without_the_filters_memory(d):
    n, nq = (1 << 17) + 333, 140
    rng = np.random.default_rng(d)
    x = rng.random((d, n), dtype=np.float32)
    ks, w, a, qqs = _batch(d, nq, rng)
    with T.Table(n, d) as t:
        t.upload(x)
        for mode in (2, 2, 0, 2, 0):
            t.set_fault_injection(mode)
            if mode == 2 and d <= 16:
                with pytest.raises(T.TopKError) as e:
                    t.query_batch(ks, w, a, qqs)
                assert e.value.status == TOPK_ERR_OOM
                continue
            ids, sc, cnt, th = t.query_batch(ks, w, a, qqs)
            assert t.last_batch_stats()["method"] == (T.BATCH_FP32 if mode == 2 else T.BATCH_BF16)
            for j in (0, 1, 63, 64, nq - 1):
                c = int(cnt[j])
                H.assert_same_result((ids[j, :c], sc[j, :c], th[j]),
                                     O.topk_numpy(x, int(ks[j]), w[j], a[j, :qqs[j]]))
        # what was built in between leaves the other calls as they are
        t.set_fault_injection(0)
        t.build_lists()
        t.build_partitions(4096, T.ORDER_KD)
        q = int(min(qqs[0], 8))
        want = O.topk_numpy(x, 50, w[0], a[0, :q])
        H.assert_same_result(t.query_ta(50, w[0], a[0, :q])[:3], want)
        H.assert_same_result(t.query_pruned(50, w[0], a[0, :q])[:3], want)
