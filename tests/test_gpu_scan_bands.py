"""Small tables with one tile per scanning CTA, k around the numbers at which its CTAs publish
28 entries each, 32, or nothing (k / CTAs of 28 and 32, 16 CTAs), against the oracle bit
for bit, with spread, equal and crowded best scores."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [15, 16, 17, 44, 100, 128])
@pytest.mark.parametrize("kind", ["uniform", "ties", "front"])
def test_k_per_cta(tiles, kind):
    n, d = 1024 * tiles - 19, 5
    rng = np.random.default_rng(tiles)
    x = rng.random((d, n), dtype=np.float32)
    if kind == "ties":
        x = np.floor(x * 6) / np.float32(8)
    elif kind == "front":
        x[:, 2000:2700] += 1
    w = (1 - rng.random(d)).astype(np.float32)
    with T.Table(n, d) as t:
        t.upload(x)
        for q in (2, 5):
            a = rng.permutation(d)[:q].astype(np.uint8)
            for k in (24 * tiles, 28 * tiles, 28 * tiles + 1, 30 * tiles, 32 * tiles, 32 * tiles + 1):
                if k <= 4096:
                    H.assert_same_result(t.query(k, w, a), O.topk_numpy(x, k, w, a))
