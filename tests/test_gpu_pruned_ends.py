"""Pruned queries whose best rows lie side by side in one partition (one CTA of the scan holds
most of the result): k at the limits of what such a CTA publishes directly, selects and
publishes, or leaves to the merge tree, on small and larger grids, with equal scores and
NaN among them, against the oracle, bit for bit."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,part_rows", [(150_001, 1024), (758_368, 8192), (3_000_017, 4096)])
@pytest.mark.parametrize("kind", ["crowd", "ties", "nan"])
@pytest.mark.parametrize("order", [T.ORDER_KD, T.ORDER_VTA])
def test_best_rows_in_one_partition(n, part_rows, kind, order):
    d = 3
    rng = np.random.default_rng([n, part_rows])
    x = rng.random((d, n), dtype=np.float32)
    crowd = rng.permutation(n)[:900]
    x[:, crowd] = 3 + x[:, crowd] * np.float32(0.01)  # one corner of the table
    if kind == "ties":
        x[:, crowd] = np.floor(x[:, crowd] * 200) / np.float32(200)
    elif kind == "nan":
        x[:, crowd[::7]] = np.nan
    w = np.array([0.7, 1.0, 0.4], np.float32)
    with T.Table(n, d) as t:
        t.upload(x)
        t.build_partitions(part_rows, order)
        for q in (1, 3):
            a = np.arange(q, dtype=np.uint8)
            for k in (16, 95, 96, 97, 191, 192, 193, 500, 767, 768, 769, 1024):
                want = O.topk_numpy(x, k, w, a)
                for _ in range(2):
                    H.assert_same_result(t.query_pruned(k, w, a)[:3], want)
