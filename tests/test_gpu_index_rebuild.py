"""Index builds written over an older one of the same handle: other orders, partition sizes
and data leave what a fresh handle builds (deterministic orders, bit for bit)."""
import numpy as np
import pytest

import topk_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 3, 4, 7, 8, 9, 17])
def test_rebuild_equals_fresh_build(d):
    n = 70001
    rng = np.random.default_rng(d)
    tables = [rng.random((d, n), dtype=np.float32) for _ in range(2)]
    tables[1][:, ::5] = np.nan
    seq = [(0, 4096, T.ORDER_KD), (0, 1024, T.ORDER_VTA), (1, 1024, T.ORDER_KD), (1, 2048, T.ORDER_PTA),
           (0, 1 << 17, T.ORDER_KD), (0, 1024, T.ORDER_VTA_THREADS), (0, 4096, T.ORDER_KD)]
    with T.Table(n, d) as t:
        at = None
        for which, rows, order in seq:
            if at != which:
                t.upload(tables[which])
                at = which
                with pytest.raises(T.TopKError):
                    t.partition_ids()  # of the data before the upload
            t.build_partitions(rows, order)
            with T.Table(n, d) as f:
                f.upload(tables[which])
                f.build_partitions(rows, order)
                assert np.array_equal(t.partition_ids(), f.partition_ids())
                for a, b in zip(t.partition_info(), f.partition_info()):
                    assert np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)
