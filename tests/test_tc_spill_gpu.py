"""Batches of more than 64 queries keep short lists on the tensor-core scan
of rows in no order; full ones spill into the query's dense run. Rows stored
cluster by cluster put all of a query's nearest in one or two lists: they
get lists that hold them whole, the CUDA-core scan's answer, and nothing
re-run while the superset is at most 64."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.hnsw import Hnsw
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu
BF16, FP8 = _lib.FV_GPU_PREC_BF16, _lib.FV_GPU_PREC_FP8


def _rows(n, dim, per, seed):
    """Integer rows, `per` consecutive ones around each centre."""
    rng = np.random.default_rng(seed)
    c = rng.integers(40, 200, (-(-n // per), dim))
    x = np.repeat(c, per, 0)[:n] + rng.integers(-9, 10, (n, dim))
    return x.astype(np.float32), rng.uniform(0, 1, (1, n)), rng


@pytest.mark.parametrize("n,dim,nq,k,prec,per", [
    (40_000, 128, 130, 33, BF16, 128), (40_000, 128, 512, 64, BF16, 100),
    (150_001, 128, 100, 64, BF16, 300), (60_000, 64, 200, 64, BF16, 5000),
    (60_000, 32, 65, 40, BF16, 128), (40_000, 200, 300, 64, BF16, 128),
    (30_000, 250, 128, 64, BF16, 90), (40_000, 128, 130, 25, 0, 128), (60_000, 96, 300, 64, 0, 200),
    (60_000, 96, 128, 200, BF16, 128), (60_000, 128, 512, 200, BF16, 60_000),
])
@pytest.mark.parametrize("share", [1.0, 0.5])
def test_rows_in_order(n, dim, nq, k, prec, per, share):
    x, cols, rng = _rows(n, dim, per, n + nq + k)
    q = x[rng.integers(0, n, nq)] + rng.integers(-2, 3, (nq, dim)).astype(np.float32)
    preds = [Cmp(0, "<", share)] * (nq - 1) + [Cmp(0, "<", 0.9)]
    gi = GpuIndex(x, cols, device=0, precision=prec)
    ids, dists, cnt, trunc = gi.brute_batch(q, preds, k)
    S, unc = _lib.lib().pv_last_superset(gi.handle), _lib.lib().pv_last_uncertain(gi.handle)
    gi.close()
    ex = GpuIndex(x, cols, device=0)
    assert _lib.lib().pv_exact_tc(ex.handle, 0) == 0
    i2, d2, c2, t2 = ex.brute_batch(q, preds, k)
    ex.close()
    assert S > 0 and (S > 64 or unc == 0)
    assert np.array_equal(cnt, c2) and np.array_equal(trunc, t2)
    assert np.array_equal(dists, d2) and np.array_equal(ids, i2)


@pytest.mark.parametrize("n,dim,nq,k,prec", [
    (150_001, 128, 130, 33, BF16), (150_001, 128, 512, 64, BF16), (80_000, 32, 65, 64, BF16),
    (150_001, 250, 100, 50, BF16), (80_000, 160, 257, 100, BF16), (150_001, 96, 512, 16, FP8),
    (150_001, 96, 100, 100, FP8),
])
@pytest.mark.parametrize("block", [0, 700])
def test_lists_spill(n, dim, nq, k, prec, block):
    """Against the shape with one group and lists of 64: the same supersets.
    `block`: consecutive rows that are one cluster, and the queries in it."""
    x, cols, rng = _rows(n, dim, 500, n + k)
    x = np.ascontiguousarray(x[rng.permutation(n)])
    if block:
        x[30_000:30_000 + block] = x[5] + rng.integers(-4, 5, (block, dim)).astype(np.float32)
    at = rng.integers(30_000, 30_000 + block, nq) if block else rng.integers(0, n, nq)
    q = x[at] + rng.integers(-2, 3, (nq, dim)).astype(np.float32)
    preds = [Cmp(0, "<", 0.5)] * (nq - 1) + [Cmp(0, "<", 0.9)]
    gi = GpuIndex(x, cols, device=0, precision=prec)
    L = _lib.lib()
    ids, dists, cnt, _ = gi.brute_batch(q, preds, k)
    unc = L.pv_last_uncertain(gi.handle)
    assert L.pv_tc_shape(gi.handle, 1, 0, 0, 0, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, preds, k)
    unc1 = L.pv_last_uncertain(gi.handle)
    gi.close()
    assert np.array_equal(cnt, c2)
    if not block:
        assert unc == 0 and unc1 == 0
    if unc == 0 and unc1 == 0 or prec != FP8:  # (re-run FP8 queries are exact)
        assert np.array_equal(ids, i2) and np.array_equal(dists, d2)


@pytest.mark.parametrize("dim,per", [(32, 100), (128, 100), (64, 4000)])
def test_builder_on_rows_in_order(dim, per):
    """The graph built behind tensor-core scans is the one built behind the
    exact FP32 scans (rows offset by a fraction refuse the former)."""
    x, _, _ = _rows(9000, dim, per, dim)
    a = Hnsw(x, 16, builder="gpu")
    b = Hnsw(x + 0.5, 16, builder="gpu")  # the same differences
    assert np.array_equal(a.l0, b.l0) and np.array_equal(a.upper, b.upper)
