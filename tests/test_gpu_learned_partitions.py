"""What the learned cut saves a pruned query, counted: on correlated data the scan that starts
from it reads fewer partitions than the scan that finds its threshold on the way.  (On
anticorrelated data it reads about as many.)  Results against the plain method, bit for bit."""
import numpy as np
import pytest

import topk_b200 as T
from tests import helpers as H

pytestmark = pytest.mark.gpu


def test_learned_cut_scans_fewer_partitions_on_correlated_data():
    n, d = 1 << 23, 8
    rng = np.random.default_rng(3)
    with T.Table(n, d) as t:
        t.generate(T.DIST_CORRELATED, 3)
        t.normalize()
        t.build_partitions(8192, T.ORDER_KD)
        t.learned_fit(n_train=4096, n_val=512, kmin=16, kmax=1024, qmin=2, qmax=d, epochs=8, miss_rate=0.02, seed=1)
        learned = plain = accepted = 0
        for _ in range(24):
            k = int(rng.integers(16, 1024))
            w = (1 - rng.random(d)).astype(np.float32)
            a = rng.permutation(d)[:int(rng.integers(2, d + 1))].astype(np.uint8)
            x, y = t.query_learned(k, w, a), t.query_pruned(k, w, a)
            H.assert_same_result(x[:3], y[:3])
            learned, plain, accepted = learned + x[3][0], plain + y[3][0], accepted + x[3][2]
        print(f"partitions scanned: learned {learned}, plain {plain}; accepted {accepted} of 24")
        assert accepted >= 20 and learned < 0.9 * plain
