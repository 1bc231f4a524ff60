"""The scan's threshold epochs and its answer by the coordinator against the oracle, bit
for bit, at the edges of what they cover: two and three tiles per CTA (no epoch, one,
several), k at the limits of the published lists, of the counting rank and of the linear
bins, and data on which the published entries cannot hold the result (equal scores, NaN,
the best rows side by side), where the merge tree answers.  And scans of several tables
that overlap on the GPU, whose CTAs may wait for places and go through the tree.
"""
import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

TILE = 1024
CTAS = 148 * 5 - 1  # scanning CTAs of a 3 <= q <= 8, small-k scan on 148 SMs


def _values(n, d, kind, seed):
    x = np.random.default_rng(seed).random((d, n), dtype=np.float32)
    if kind == "ties":
        x = np.floor(x * 3) / np.float32(4)
    elif kind == "nan":
        x[:, ::3] = np.nan
    elif kind == "few":  # fewer numbers than most k
        keep = x[:, :700].copy()
        x[:] = np.nan
        x[:, n // 2:n // 2 + 700] = keep
    elif kind == "front":  # the best rows side by side, at the front of one tile
        x[:, 5000:5600] += 2
    elif kind == "rising":
        x += np.linspace(0, 4, n, dtype=np.float32)
    elif kind == "falling":
        x -= np.linspace(0, 4, n, dtype=np.float32)
    return x


@pytest.mark.parametrize("n", [2 * TILE + 1, CTAS * TILE, 2 * CTAS * TILE, 2 * CTAS * TILE + 1, 5 * CTAS * TILE - 3])
@pytest.mark.parametrize("kind", ["uniform", "ties", "nan", "few", "front", "rising", "falling"])
def test_epochs_and_answers(n, kind):
    d = 4
    x = _values(n, d, kind, n % 97)
    rng = np.random.default_rng(5)
    with T.Table(n, d) as t:
        t.upload(x)
        for q in (1, 2, 3):
            w = (1 - rng.random(d)).astype(np.float32)
            a = rng.permutation(d)[:q].astype(np.uint8)
            for k in (1, 32, 33, 97, 184, 185, 186, 257, 1024, 4096):
                H.assert_same_result(t.query(k, w, a), O.topk_numpy(x, k, w, a))


@pytest.mark.parametrize("lo,hi", [(0, 2500), (3, 1024 * 900 + 5), (77, 1024 * 2300 - 1)])
def test_row_ranges(lo, hi):
    n, d = 1024 * 2300, 3
    x = _values(n, d, "uniform", 3)
    w, a = np.array([0.5, -0.7, 0.9], np.float32), np.array([2, 0, 1], np.uint8)
    with T.Table(n, d) as t:
        t.upload(x)
        for k in (5, 100, 1000):
            H.assert_same_result(t.query(k, w, a, lo, hi), O.topk_numpy(x, k, w, a, lo, hi))


def test_overlapping_scans_of_several_tables():
    """Four tables, each with its own stream and scratch: scans that fill the GPU several
    times over, so CTAs of one wait for places that the others hold."""
    torch = pytest.importorskip("torch")
    d, ks = 8, (16, 300, 1024, 4000)
    tables, want, got = [], [], []
    rng = np.random.default_rng(11)
    for j in range(4):
        x = _values(3_000_000 + 1717 * j, d, ("uniform", "ties", "front", "uniform")[j], j)
        t = T.Table(x.shape[1], d)
        t.upload(x)
        tables.append(t)
        queries = [(k, (1 - rng.random(d)).astype(np.float32), rng.permutation(d)[:q].astype(np.uint8))
                   for k in ks for q in (1, 2, 5, 8)]
        want.append([O.topk_numpy(x, *qr) for qr in queries])
        got.append([(torch.zeros(qr[0], dtype=torch.int64, device="cuda"), torch.zeros(qr[0], device="cuda"), qr)
                    for qr in queries])
    streams = [torch.cuda.Stream() for _ in tables]
    torch.cuda.synchronize()
    for _ in range(2):
        for i in range(len(got[0])):
            for t, s, g in zip(tables, streams, got):
                ids, sc, (k, w, a) = g[i]
                t.query_device(k, w, a, ids.data_ptr(), sc.data_ptr(), stream=s.cuda_stream)
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        for (ids, sc, _), (wi, ws, _) in zip(g, w):
            assert np.array_equal(ids.cpu().numpy().astype(np.uint64), wi)
            assert np.array_equal(sc.cpu().numpy().view(np.uint32), ws.view(np.uint32))
    for t in tables:
        t.close()
