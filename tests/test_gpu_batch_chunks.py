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


@pytest.mark.parametrize("d", [17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("n,method", [((1 << 17) - 1, T.BATCH_FP32), (1 << 17, T.BATCH_BF16),
                                      ((1 << 17) + 300, T.BATCH_BF16)])
def test_wide_tables_on_the_filter(d, n, method):
    """Two to four K blocks of the tensor-core filter, from the row count it starts at; more
    query tiles than one CTA takes; attributes repeated and in any order, signed weights."""
    rng = np.random.default_rng([d, n])
    x = rng.uniform(-1, 1, (d, n)).astype(np.float32)
    nq = 7 * 128 + 1
    ks = rng.integers(1, 300, nq).astype(np.uint64)
    qqs = rng.integers(1, 32, nq, endpoint=True).astype(np.uint32)
    w = rng.uniform(-1, 1, (nq, d)).astype(np.float32)
    a = rng.integers(0, d, (nq, 32)).astype(np.uint8)
    a[0, :2] = d - 1, 0  # the ends of the K blocks
    with T.Table(n, d) as t:
        t.upload(x)
        ids, sc, cnt, th = t.query_batch(ks, w, a, qqs)
        st = t.last_batch_stats()
    assert st["method"] == method
    if method == T.BATCH_BF16:
        assert st["max_err_ratio"] < 0.5
    for j in (0, 1, 127, 128, 500, nq - 1):
        c = int(cnt[j])
        H.assert_same_result((ids[j, :c], sc[j, :c], th[j]), O.topk_numpy(x, int(ks[j]), w[j], a[j, :qqs[j]]))


def test_wide_table_learned_start_on_the_filter():
    n, d = (1 << 17) + 5000, 20
    rng = np.random.default_rng(4)
    x = rng.random((d, n), dtype=np.float32)
    with T.Table(n, d) as t:
        t.upload(x)
        t.build_partitions(4096, T.ORDER_KD)
        t.learned_fit(1024, 256, kmin=4, kmax=128, epochs=5)
        t.set_batch_method(T.BATCH_LEARNED)
        nq = 140
        ks = rng.integers(4, 128, nq).astype(np.uint64)
        w = (1 - rng.random((nq, d))).astype(np.float32)
        a = rng.permuted(np.tile(np.arange(d, dtype=np.uint8), (nq, 1)), axis=1)
        qqs = rng.integers(2, d, nq, endpoint=True).astype(np.uint32)
        ids, sc, cnt, th = t.query_batch(ks, w, a, qqs)
        assert t.last_batch_stats()["method"] == T.BATCH_LEARNED
    for j in range(0, nq, 13):
        c = int(cnt[j])
        H.assert_same_result((ids[j, :c], sc[j, :c], th[j]), O.topk_numpy(x, int(ks[j]), w[j], a[j, :qqs[j]]))
