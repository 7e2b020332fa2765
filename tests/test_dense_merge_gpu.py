"""Merges of more than 32 keys: the radix select over the keys' own range, at
list lengths around its limits; many equal distances (the row decides) and
supersets that are re-ranked. Exact ids against the CUDA-core scan's."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 32, 33, 64, 65, 127, 128, 129, 256, 257, 511, 1000])
@pytest.mark.parametrize("values", ["ties", "spread"])
def test_ids_in_order(k, values):
    rng = np.random.default_rng(k)
    n, dim, nq = 30_011, 64, 40
    x = rng.integers(0, 2 if values == "ties" else 256, (n, dim)).astype(np.float32)
    q = rng.integers(0, 2 if values == "ties" else 256, (nq, dim)).astype(np.float32)
    q[1] = x[7]  # a distance of zero
    cols = rng.uniform(0, 1, (1, n))
    # shares that pass: all, few more than k, fewer than k, none
    cuts = [1.0, (k + 8) / n, k / 2 / n, 0.0]
    preds = [Cmp(0, "<", cuts[i % 4]) for i in range(nq)]
    gi = GpuIndex(x, cols, device=0, precision=_lib.FV_GPU_PREC_BF16)
    ids, dists, cnt, trunc = gi.brute_batch(q, preds, k)
    assert _lib.lib().pv_last_superset(gi.handle) == k  # no re-rank
    gi.close()
    d = (q * q).sum(1)[:, None] + (x * x).sum(1)[None] - 2 * (q @ x.T)  # whole numbers
    for i in range(nq):
        rows = np.flatnonzero(cols[0] < cuts[i % 4])
        want = rows[np.lexsort((rows, d[i, rows]))][:k]
        assert cnt[i] == len(want) and trunc[i] == (len(rows) > k)
        assert np.array_equal(ids[i, :cnt[i]].astype(np.int64), want)
        assert np.array_equal(dists[i, :cnt[i]], d[i, want])


@pytest.mark.parametrize("k", [9, 16, 17, 64, 200])
@pytest.mark.parametrize("dim", [32, 100, 128])
def test_superset_in_any_order(k, dim):
    """Real-valued rows: the re-ranked answers of the exact mode."""
    rng = np.random.default_rng(k + dim)
    n, nq = 40_003, 70
    x = rng.standard_normal((n, dim)).astype(np.float32)
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    cols = rng.uniform(0, 1, (1, n))
    preds = [Cmp(0, "<", [1.0, 0.01, 0.0001][i % 3]) for i in range(nq)]
    gi = GpuIndex(x, cols, device=0)
    ids, dists, cnt, _ = gi.brute_batch(q, preds, k)
    assert _lib.lib().pv_last_exact_tc(gi.handle) == 1
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, preds, k)
    gi.close()
    assert np.array_equal(cnt, c2)
    np.testing.assert_allclose(dists, d2, rtol=2e-6)
    for i in range(nq):
        assert len(set(ids[i, :cnt[i]].tolist())) == cnt[i]
        assert np.all(np.diff(dists[i, :cnt[i]]) >= 0)
