"""Performance cases of topk_b200: what a user of the library has it do, by size.

Each case is one pass through the public Python entry points (`topk_b200.Table`) over
tables of the shapes the benchmark, the tests and the reference's harness use: single
exact top-k queries (synchronous and on a stream), batches, pruned queries, the
threshold algorithm, index builds and table files.  Small tables are made with torch
from the seed and uploaded; tables above 1 GB come from the library's own seeded
generator, which fills device memory.
"""
import math
import os
import tempfile

import numpy as np
import torch

import topk_b200 as T

DISTS = {"independent": T.DIST_INDEPENDENT, "correlated": T.DIST_CORRELATED,
         "anticorrelated": T.DIST_ANTICORRELATED, "mixed": T.DIST_MIXED}
ORDERS = {"kd": T.ORDER_KD, "vta": T.ORDER_VTA, "pta": T.ORDER_PTA}
UPLOAD_BYTES = 1 << 30  # larger tables are generated on the device
EXACT_OPS = 4e11          # multiply-adds above which no 64-bit answer is computed


def listed():
    return [
        # The reference's own small configuration: one query over 2^20 x 8, where the
        # launch, the end of the scan and the host call are most of the time.
        {"name": "query-1m", "kind": "query", "n": 1 << 20, "d": 8, "q": 4, "k": 16, "dist": "independent",
         "neg": False},
        # An ordinary table with odd sizes, an odd attribute count and weights of both signs.
        {"name": "query-10m-ragged", "kind": "query", "n": 10_000_019, "d": 13, "q": 5, "k": 100,
         "dist": "correlated", "neg": True},
        # The headline table (2^28 x 16): one synchronous query of the benchmark's mix.
        {"name": "query-268m", "kind": "query", "n": 1 << 28, "d": 16, "q": 8, "k": 256, "dist": "independent",
         "neg": False},
        # The benchmark's 16-query step (q in {2, 4, 8, 16} x k in {16, 64, 256, 1024}) issued
        # on a stream into device buffers, as a program with its own pipeline does.
        {"name": "stream-16-queries", "kind": "stream", "n": 1 << 24, "d": 16, "dist": "independent", "neg": False},
        # A small service: a hundred requests at once over a table of 200 thousand rows.
        {"name": "batch-100-small", "kind": "batch", "n": 200_003, "d": 8, "nq": 100, "kmax": 100,
         "dist": "independent", "neg": False, "keep": False},
        # A table wider than 16 attributes: the batch runs on the exact FP32 scorer.
        {"name": "batch-300-wide", "kind": "batch", "n": 2_000_003, "d": 24, "nq": 300, "kmax": 256,
         "dist": "anticorrelated", "neg": True, "keep": False},
        # The benchmark's batch: 4096 queries over 2^26 x 16, result arrays kept by the caller.
        {"name": "batch-4096", "kind": "batch", "n": 1 << 26, "d": 16, "nq": 4096, "kmax": 1024,
         "dist": "independent", "neg": False, "keep": True},
        # The benchmark's pruned query: 2^27 x 8 anticorrelated rows in 2048 kd partitions.
        {"name": "pruned-134m", "kind": "pruned", "n": 1 << 27, "d": 8, "q": 4, "k": 128, "dist": "anticorrelated",
         "part_rows": 1 << 16, "order": "kd", "neg": False},
        # The threshold algorithm over sorted lists, on the data it is meant for.
        {"name": "ta-4m", "kind": "ta", "n": 1 << 22, "d": 8, "q": 4, "k": 64, "dist": "correlated", "neg": False},
        # Building the pruning index of a table (once per table), read back whole.
        {"name": "index-kd-6m", "kind": "index", "n": 6_000_011, "d": 8, "dist": "anticorrelated",
         "part_rows": 1 << 12, "order": "kd"},
        # A table file to a first answer: CSV parsed, attributes normalised, one query.
        {"name": "csv-to-answer", "kind": "csv", "n": 500_003, "d": 8, "q": 4, "k": 16, "dist": "independent",
         "neg": False},
        # SLA's index: the skyline layer of every row, at the sizes the reference's SLA serves.
        {"name": "skyline-30k", "kind": "skyline", "n": 30_011, "d": 4, "dist": "anticorrelated"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["query", "stream", "batch", "pruned", "ta", "index", "csv", "skyline"],
                       [6, 2, 4, 3, 1, 1, 1, 1])[0]
    dist = rng.choice(["independent", "correlated", "anticorrelated"])
    neg = rng.random() < 0.3
    if kind == "query":
        d = rng.randint(2, 24)
        n = _log_int(rng, 1000, min(1 << 28, (1 << 32) // d))
        return {"kind": kind, "n": n, "d": d, "q": rng.randint(1, d), "k": _log_int(rng, 1, 4096), "dist": dist,
                "neg": neg}
    if kind == "stream":
        return {"kind": kind, "n": _log_int(rng, 100_000, 1 << 25), "d": 16, "dist": dist, "neg": neg}
    if kind == "batch":
        d = rng.randint(2, 24)
        nq = _log_int(rng, 8, 4096)
        pairs = (1 << 32) if d > 16 else (1 << 35)  # (query, row) pairs: wide tables take the FP32 scorer
        n = _log_int(rng, 20_000, min(1 << 25, pairs // nq))
        return {"kind": kind, "n": n, "d": d, "nq": nq, "kmax": _log_int(rng, 16, 1024), "dist": dist, "neg": neg,
                "keep": rng.random() < 0.5}
    if kind == "pruned":
        d = rng.randint(3, 8)
        n = _log_int(rng, 500_000, 1 << 26)
        return {"kind": kind, "n": n, "d": d, "q": rng.randint(2, d), "k": _log_int(rng, 16, 1024), "dist": dist,
                "part_rows": 1 << rng.randint(12, 15), "order": rng.choice(sorted(ORDERS)), "neg": neg}
    if kind == "ta":
        d = rng.randint(2, 8)
        return {"kind": kind, "n": _log_int(rng, 50_000, 1 << 23), "d": d, "q": rng.randint(2, d),
                "k": _log_int(rng, 16, 1024), "dist": rng.choice(["correlated", "independent"]), "neg": neg}
    if kind == "index":
        return {"kind": kind, "n": _log_int(rng, 200_000, 6_000_011), "d": rng.randint(2, 8), "dist": dist,
                "part_rows": 1 << rng.randint(11, 14), "order": rng.choice(sorted(ORDERS))}
    if kind == "csv":
        d = rng.randint(2, 16)
        return {"kind": kind, "n": _log_int(rng, 20_000, 4_000_000 // d), "d": d, "q": rng.randint(1, d),
                "k": _log_int(rng, 1, 1024), "dist": dist, "neg": neg}
    return {"kind": kind, "n": _log_int(rng, 2000, 30_011), "d": rng.randint(2, 4), "dist": dist}


def _uploads(case):
    return 4 * case["n"] * case["d"] <= UPLOAD_BYTES


def _values(case, seed):
    """(d, n) float32 values in [0, 1] on the GPU, of the harness's three distributions,
    each column stretched to [0, 1] as its normalisation does."""
    n, d = case["n"], case["d"]
    g = torch.Generator("cuda").manual_seed(1_000_003 * seed + 17)
    if case["dist"] == "correlated":
        x = torch.rand(n, generator=g, device="cuda") + 0.05 * torch.randn(d, n, generator=g, device="cuda")
    elif case["dist"] == "anticorrelated":
        x = torch.rand(d, n, generator=g, device="cuda").clamp_(min=1e-7).log_().neg_()
        x.mul_(0.5 * d / x.sum(0))
        x.add_(torch.randn(d, n, generator=g, device="cuda"), alpha=0.05)
    else:
        x = torch.rand(d, n, generator=g, device="cuda")
    lo, hi = x.min(1, keepdim=True).values, x.max(1, keepdim=True).values
    return x.sub_(lo).div_(hi - lo).clamp_(0.0, 1.0)


def _table(case, seed):
    t = T.Table(case["n"], case["d"])
    if _uploads(case):
        t.upload(_values(case, seed).cpu().numpy())
    else:
        t.generate(DISTS[case["dist"]], seed)
        t.normalize()
    return t


def _weights(rng, shape, neg):
    w = 1.0 - rng.random(shape, dtype=np.float32)  # (0, 1]
    return np.where(rng.random(shape) < 0.3, -w, w).astype(np.float32) if neg else w


def _single(case, seed):
    """Weights by attribute id and the q queried attributes in summation order."""
    rng = np.random.default_rng([seed, 1])
    return _weights(rng, case["d"], case["neg"]), rng.permutation(case["d"])[:case["q"]].astype(np.uint8)


def _stream_queries(case, seed):
    rng = np.random.default_rng([seed, 2])
    d = case["d"]
    return [(k, _weights(rng, d, case["neg"]), np.arange(d - q, d, dtype=np.uint8))
            for q in (2, 4, 8, 16) for k in (16, 64, 256, 1024)]


def _batch_queries(case, seed):
    rng = np.random.default_rng([seed, 3])
    nq, d = case["nq"], case["d"]
    ks = rng.integers(1, case["kmax"], nq, endpoint=True).astype(np.uint64)
    ks[0] = case["kmax"]  # the width of the result arrays
    qqs = rng.integers(min(2, d), d, nq, endpoint=True).astype(np.uint32)
    attrs = rng.permuted(np.tile(np.arange(d, dtype=np.uint8), (nq, 1)), axis=1)
    return ks, _weights(rng, (nq, d), case["neg"]), attrs, qqs


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "csv":
        s["dir"] = tempfile.TemporaryDirectory()
        s["path"] = os.path.join(s["dir"].name, "table.csv")
        with _table(case, seed) as t:
            t.save_csv(s["path"])
        s["table"] = T.Table(case["n"], case["d"])
        s["query"] = _single(case, seed)
        return s
    s["table"] = t = _table(case, seed)
    if kind in ("query", "pruned", "ta"):
        s["query"] = _single(case, seed)
    if kind == "pruned":
        t.build_partitions(case["part_rows"], ORDERS[case["order"]])
    elif kind == "ta":
        t.build_lists()
    elif kind == "stream":
        s["queries"] = _stream_queries(case, seed)
        s["ids"] = [torch.zeros(min(k, case["n"]), dtype=torch.int64, device="cuda") for k, _, _ in s["queries"]]
        s["scores"] = [torch.zeros(min(k, case["n"]), device="cuda") for k, _, _ in s["queries"]]
        s["stream"] = torch.cuda.current_stream().cuda_stream
    elif kind == "batch":
        s["queries"] = ks, _, _, _ = _batch_queries(case, seed)
        if case["keep"]:
            nq, kstride = case["nq"], int(min(ks.max(), case["n"]))
            s["out"] = (np.zeros((nq, kstride), np.uint64), np.zeros((nq, kstride), np.float32),
                        np.zeros(nq, np.uint64), np.zeros(nq, np.float32))
    return s


def run(s):
    kind, t, case = s["kind"], s["table"], s["case"]
    if kind == "query":
        return t.query(case["k"], *s["query"])
    if kind == "stream":
        for (k, w, a), ids, sc in zip(s["queries"], s["ids"], s["scores"]):
            t.query_device(k, w, a, ids.data_ptr(), sc.data_ptr(), stream=s["stream"])
        return s["ids"], s["scores"]
    if kind == "batch":
        ks, w, a, qqs = s["queries"]
        return t.query_batch(ks, w, a, qqs, out=s.get("out"))
    if kind == "pruned":
        return t.query_pruned(case["k"], *s["query"])[:3]  # the statistics depend on timing
    if kind == "ta":
        return t.query_ta(case["k"], *s["query"])
    if kind == "index":
        t.build_partitions(case["part_rows"], ORDERS[case["order"]])
        return (t.partition_ids(),) + t.partition_info()
    if kind == "csv":
        t.load_csv(s["path"])
        mins, maxs = t.normalize()
        return (mins, maxs) + t.query(case["k"], *s["query"])
    return t.skyline_layers()


def work(case):
    kind, n, d = case["kind"], case["n"], case["d"]
    if kind in ("query", "pruned", "ta"):
        q, k = case["q"], min(case["k"], n)
        if kind == "query":
            return {"bytes": 4 * n * q + 12 * k, "flops": 2 * n * q}
        # what an index can leave: the k winners' values (and their list entries)
        per = 4 * q + 12 + (8 if kind == "ta" else 0)
        return {"bytes": per * k, "flops": 2 * q * k}
    if kind == "stream":
        return {"bytes": sum(4 * (4 * n * q) + 12 * (16 + 64 + 256 + 1024) for q in (2, 4, 8, 16)),
                "flops": sum(4 * 2 * n * q for q in (2, 4, 8, 16))}
    if kind == "batch":
        nq, q = case["nq"], (min(2, d) + d) / 2
        return {"bytes": 4 * n * d + nq * (5 * d + 12) + 6 * nq * case["kmax"], "flops": 2 * nq * n * q}
    if kind == "index":
        parts = -(-n // case["part_rows"])
        return {"bytes": 8 * n * d + 4 * n + 12 * parts * d, "flops": 3 * n * d}
    if kind == "csv":
        return {"bytes": (9 + 4 + 8) * n * d + 4 * n * case["q"], "flops": 2 * n * case["q"] + 2 * n * d}
    return {"bytes": 4 * n * d + 4 * n, "flops": n * d}


def _top(table, w, attr, k):
    """The k best 64-bit scores, ascending; table: (d, n) float64."""
    s = torch.zeros(table.shape[1], dtype=torch.float64, device=table.device)
    for a in attr:
        s += table[int(a)] * float(w[int(a)])
    return torch.topk(s, min(int(k), len(s))).values.flip(0).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("index", "skyline") or not _uploads(case):
        return None
    if kind == "batch" and case["nq"] * case["n"] * case["d"] > EXACT_OPS:
        return None
    x = _values(case, seed).double()
    if kind == "csv":
        # the file holds 6 decimals, read back as FP32; then (v - min) / (max - min) with
        # the reference's starting values (max from 0)
        x = x.mul(1e6).round().div(1e6).float().double()
        lo, hi = x.min(1).values, x.max(1).values.clamp(min=0.0)
        norm = (x - lo[:, None]) / (hi - lo)[:, None]
        top = _top(norm, *_single(case, seed), case["k"])
        return lo.cpu().numpy(), hi.cpu().numpy(), None, top, float(top[0])
    if kind == "stream":
        return (None, [_top(x, w, a, k) for k, w, a in _stream_queries(case, seed)])
    if kind == "batch":
        ks, w, a, qqs = _batch_queries(case, seed)
        scores = np.zeros((case["nq"], int(min(ks.max(), case["n"]))))
        ths = np.zeros(case["nq"])
        for j in range(case["nq"]):
            top = _top(x, w[j], a[j, :qqs[j]], ks[j])
            scores[j, :len(top)] = top
            ths[j] = top[0]
        return None, scores, None, ths
    top = _top(x, *_single(case, seed), case["k"])
    return (None, top, float(top[0])) + ((None,) if kind == "ta" else ())
