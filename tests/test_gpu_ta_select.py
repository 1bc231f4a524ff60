"""GPU: the selection of the threshold algorithm where its bins or its list can fail.

Exact results (bit for bit) at k around the block's list of 4096 keys, with every score
equal (one bin, more keys than the list), scores of a few values, ranges that are not
finite or that a few objects stretch, and walks of several blocks that carry their best.
"""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _values(kind, n, d, rng):
    x = rng.random((d, n), dtype=np.float32)
    if kind == "equal":
        x[:] = 0.5
    elif kind == "few":
        x = np.floor(x * 3) / 3
    elif kind == "outliers":
        x[:, rng.integers(0, n, 5)] = 1e30
    elif kind == "infinite":
        x *= 3e38
        x[:, rng.integers(0, n, 9)] = np.inf
    elif kind == "correlated":
        x = rng.random((1, n), dtype=np.float32) * 0.9 + x * 0.1
    return np.ascontiguousarray(x, dtype=np.float32)


@pytest.mark.parametrize("kind", ["uniform", "equal", "few", "outliers", "infinite", "correlated"])
@pytest.mark.parametrize("n", [1, 2049, 100003])
def test_ta_selection(kind, n):
    d = 4
    rng = np.random.default_rng(n)
    x = _values(kind, n, d, rng)
    with T.Table(n, d) as t:
        t.upload(x)
        t.build_lists()
        for k in (1, 64, 2048, 4095, 4096):
            for w in (np.array([0.25, 1.0, 0.5, 0.125], np.float32), np.array([0.25, -1.0, 0.5, 0.0], np.float32)):
                if kind == "infinite" and w.min() <= 0:
                    continue  # inf - inf
                for a in ([0, 1, 2, 3], [2, 2, 0], [3]):
                    a = np.array(a, np.uint8)
                    H.assert_same_result(t.query_ta(k, w, a)[:3], O.topk_numpy(x, k, w, a))
