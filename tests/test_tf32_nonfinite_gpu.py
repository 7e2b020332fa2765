"""Exact batches over rows and queries that hold infinities, NaN or values
whose squares leave the f32 range: the answers are those of the CUDA-core
scan, filters that pass fewer rows than the re-ranked superset included."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu
N, NQ, K = 20_003, 24, 10


def both_routes(x, cols, q, preds, k, prec=0):
    gi = GpuIndex(x, cols, device=0, precision=prec)
    got = gi.brute_batch(q, preds, k)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    want = gi.brute_batch(q, preds, k)
    gi.close()
    return got, want


def same(got, want):
    ids, dists, cnt, trunc = got
    i2, d2, c2, t2 = want
    assert np.array_equal(cnt, c2) and np.array_equal(trunc, t2)
    for i, c in enumerate(cnt):
        assert np.array_equal(ids[i, :c], i2[i, :c]), i
        np.testing.assert_array_equal(dists[i, :c], d2[i, :c])


@pytest.mark.parametrize("dim", [64, 128, 200, 384])
@pytest.mark.parametrize("where,value", [
    ("rows", np.inf), ("rows", -np.inf), ("rows", np.nan), ("rows", 1e20), ("rows", -3e38),
    ("query", np.inf), ("query", np.nan), ("query", 1e20), ("both", np.inf), ("both", 1e20),
])
def test_values_without_a_finite_square(dim, where, value):
    rng = np.random.default_rng(dim)
    # multiples of a quarter up to 16: every f32 sum is exact in any order
    x = (rng.integers(-64, 65, (N, dim)) / 4).astype(np.float32)
    q = (rng.integers(-64, 65, (NQ, dim)) / 4).astype(np.float32)
    order = rng.permutation(N)
    cols = np.empty((1, N))
    cols[0, order] = np.arange(N)
    bad = order[[0, 3, 7, 900]]  # among the first rows of every filter, one beyond the small ones
    if where != "query":
        x[bad, rng.integers(0, dim, 4)] = value
    if where != "rows":
        q[[1, 2, 6, 11], rng.integers(0, dim, 4)] = value
    # of every query's own filter: fewer rows than k, than the superset of 4k, and more
    pass_rows = [6, 20, 39, 40, 41, 200, 5000, N]
    preds = [Cmp(0, "<", float(pass_rows[i % 8])) for i in range(NQ)]
    same(*both_routes(x, cols, q, preds, K))


@pytest.mark.parametrize("dim,m", [(128, 2220), (200, 1776)])
def test_norms_whose_sum_overflows(dim, m):
    """||x||^2 and ||q||^2 are finite, their sum is not, and the nearest row
    (the query itself) is among those the norm form puts at infinity. Every
    value is a TF32 value."""
    rng = np.random.default_rng(dim)
    signs = rng.choice([-1.0, 1.0], dim)
    x = np.zeros((4000, dim), np.float32)
    lengths = np.arange(m // 2, m * 4 // 5)
    at = rng.permutation(4000)[:len(lengths) + 1]
    x[at[1:]] = (lengths[:, None] * 2.0 ** 49) * signs
    x[at[0]] = m * 2.0 ** 49 * signs
    q = np.repeat(x[at[:1]], 16, 0)
    assert np.isfinite((q[0] ** 2).sum(dtype=np.float32))
    got, want = both_routes(x, None, q, [None] * 16, K)
    assert want[0][0, 0] == at[0] and want[1][0, 0] == 0
    same(got, want)


def test_wide_bf16_upload():
    """Rows too wide for the BF16 scan are answered from the f32 rows."""
    rng = np.random.default_rng(3)
    x = (rng.integers(-64, 65, (N, 300)) / 4).astype(np.float32)
    q = (rng.integers(-64, 65, (NQ, 300)) / 4).astype(np.float32)
    cols = np.arange(N, dtype=np.float64)[None]
    x[3, 5], x[8, 7] = np.nan, np.inf
    same(*both_routes(x, cols, q, [Cmp(0, "<", 15.0 + i) for i in range(NQ)], K,
                      _lib.FV_GPU_PREC_BF16))
