"""k above 2048 on a table with many rows at the best score, one tile per scanning CTA:
about 93 tied entries of each CTA are published, more than the coordinator reads when it
bounds the k-th best, so how many reach its bound depends on the order in which the CTAs
arrived.  Several queries each, with a cold L2 (which mixes that order), against the
oracle, bit for bit."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2049, 2304, 2560, 3072, 4095, 4096])
@pytest.mark.parametrize("q", [3, 8])
def test_more_ties_than_the_bound_reads(k, q):
    torch = pytest.importorskip("torch")
    n, d = 302_080, 8
    x = np.random.default_rng(k).random((d, n), dtype=np.float32)
    x[:, ::11] = 1
    w, a = np.ones(d, np.float32), np.arange(q, dtype=np.uint8)
    want = O.topk_numpy(x, k, w, a)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    with T.Table(n, d) as t:
        t.upload(x)
        for r in range(60):
            flush.fill_(r)
            torch.cuda.synchronize()
            H.assert_same_result(t.query(k, w, a), want)
