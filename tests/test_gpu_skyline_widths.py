"""Skyline layers at the widths and row counts where the step kernel's forms change (padded
to 1, 2, 4, 8, 16 and 32 values; blocks of 256 rows; chains through a block) against the
peeling of the oracle."""
import numpy as np
import pytest

import topk_b200 as T
from oracle import sla_oracle as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 5, 9, 17])
@pytest.mark.parametrize("n", [101, 256, 257, 400])
@pytest.mark.parametrize("kind", ["uniform", "coarse", "chain"])
def test_layers(d, n, kind):
    x = np.random.default_rng([d, n]).random((d, n), dtype=np.float32)
    if kind == "coarse":
        x = np.floor(x * 4) / np.float32(4)
    elif kind == "chain":  # every row dominates the next: depths up to n
        x = np.tile(np.linspace(1, 0, n, dtype=np.float32), (d, 1))
    with T.Table(n, d) as t:
        t.upload(np.ascontiguousarray(x))
        layers, count = t.skyline_layers()
    want = S.skyline_layers(x)
    assert np.array_equal(layers.astype(np.int64), want) and count == int(want.max()) + 1
