"""Tied scores where the scan's coordinator bounds the k-th best by id, against the oracle
bit for bit: many rows share the best score, a dense run of them first in the table (their
ids are the largest ~ids, at the top of the 32-bit range) and the rest spread thinly."""
import ctypes as C

import numpy as np
import pytest

import topk_b200 as T
from oracle import oracle as O
from topk_b200 import _lib
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _zero_one(n, run, step):
    """One 0/1 column: ones in rows [0, run) and in every step-th row."""
    x = np.zeros((1, n), np.float32)
    x[0, :run] = 1
    x[0, ::step] = 1
    return x


# one tile per scanning CTA (no threshold epoch) in the first three, several epochs in the last
@pytest.mark.parametrize("n", [200_003, 400_000, 700_001, 3_000_017])
@pytest.mark.parametrize("run,step", [(80, 180), (40, 97), (95, 411), (300, 233)])
def test_dense_run_of_ties_at_row_0(n, run, step):
    torch = pytest.importorskip("torch")
    L = T.load()
    x = _zero_one(n, run, step)
    w, a = np.ones(1, np.float32), np.zeros(1, np.uint8)
    stream = torch.cuda.current_stream().cuda_stream
    ld = (n + 63) // 64 * 64
    dt = torch.zeros(ld, device="cuda")
    dt[:n] = torch.from_numpy(x[0]).cuda()
    th = torch.empty(1, device="cuda")
    with T.Table(n, 1) as t:
        t.upload(x)
        for k in (8, 12, 16, 20, 24, 32, 100, 300, 1000):
            want = O.topk_numpy(x, k, w, a)
            H.assert_same_result(t.query(k, w, a), want)
            for noalloc in (False, True):
                ids = torch.full((k,), -1, dtype=torch.int64, device="cuda")
                sc = torch.full((k,), -1.0, device="cuda")
                if noalloc:
                    st = L.topk_query_noalloc(C.c_void_p(dt.data_ptr()), n, ld, 1, k, 1, w, a,
                                              C.c_void_p(ids.data_ptr()), C.c_void_p(sc.data_ptr()),
                                              C.c_void_p(th.data_ptr()), C.c_void_p(stream))
                    assert st == _lib.OK, L.topk_last_error()
                else:
                    t.query_device(k, w, a, ids.data_ptr(), sc.data_ptr(), stream=stream)
                torch.cuda.synchronize()
                assert np.array_equal(ids.cpu().numpy().astype(np.uint64), want[0]), (k, noalloc)
                assert np.array_equal(sc.cpu().numpy(), want[1])
        t.build_partitions(1024)
        for k in (8, 16, 32, 300):
            H.assert_same_result(t.query_pruned(k, w, a)[:3], O.topk_numpy(x, k, w, a))
