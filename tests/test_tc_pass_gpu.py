"""The tensor-core pass at the edges of its shapes (query replicas, one to
three epilogue groups, lists that fill), and its estimated admission bound."""
import ctypes as C

import numpy as np
import pytest

from oracle import cpu
from paves_b200 import _lib, datagen, pred
from paves_b200.index import GpuIndex
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu


def check(gi, x, cols, q, preds, k):
    bp = pred.concat(preds, len(x))
    ids, dists, cnt, _ = gi.brute_batch_raw(q, bp, k)
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q, bp, k)
    for i in range(len(q)):
        n = int(o_cnt[i])
        assert cnt[i] == n
        assert np.array_equal(ids[i, :n], o_ids[i, :n].astype(np.uint64)), i
        assert np.array_equal(dists[i, :n], o_d[i, :n]), i


@pytest.mark.parametrize("nq,k,n", [
    (1, 1, 5000), (32, 10, 5000), (33, 10, 5001), (64, 64, 4999), (65, 48, 3000), (65, 49, 3000),
    (128, 64, 3001), (129, 100, 2600), (300, 10, 200_000), (70, 100, 200_000),
])
@pytest.mark.parametrize("prec", [_lib.FV_GPU_PREC_BF16, _lib.FV_GPU_PREC_FP32])
def test_exact_on_integers(nq, k, n, prec):
    # BF16 rows (certified exact), and the f32 rows read as TF32 (16+ queries)
    ds = datagen.make_dataset(n, 64, nq=nq)
    gi = GpuIndex(ds.vectors, ds.cols, device=0, precision=prec)
    preds = [None if i % 3 == 0 else Cmp(datagen.COL_PRICE, "<", 30.0 * (1 + i % 30))
             for i in range(nq)]
    check(gi, ds.vectors, ds.cols, ds.queries, preds, k)
    gi.close()


def test_estimated_bound_too_low_is_re_run():
    # 160,000 rows, 64 queries: 148 ranges of 8 tiles, of which the sample
    # takes every other; 384 rows near the queries fill three of its tiles, so
    # its bound lets through fewer rows than the superset of 400 wants
    n, dim, k = 160_000, 16, 100
    rng = np.random.default_rng(3)
    x = rng.integers(100, 200, (n, dim)).astype(np.float32)
    for tile in (0, 2, 4):
        x[tile * 128:(tile + 1) * 128] = rng.integers(0, 4, (128, dim))
    q = rng.integers(0, 4, (64, dim)).astype(np.float32)
    cols = np.zeros((1, n))
    gi = GpuIndex(x, cols, device=0, precision=_lib.FV_GPU_PREC_FP8)
    check(gi, x, cols, q, [None] * 64, k)
    assert _lib.lib().pv_last_uncertain(gi.handle) == 64
    gi.close()
