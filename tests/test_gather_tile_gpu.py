"""Selective filters shared by a batch: the tiled distances of the listed rows
(12 queries and more) and merges of long runs, against the oracle."""
import numpy as np
import pytest

from oracle import cpu
from paves_b200 import _lib, pred
from paves_b200.index import GpuIndex
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,dim,rows,k", [
    (11, 128, 100, 10), (12, 128, 63, 10), (64, 128, 64, 64), (65, 128, 65, 33), (64, 100, 4000, 10),
    (130, 132, 1500, 32), (20, 512, 1600, 5), (33, 3, 1536, 64), (16, 260, 1537, 1), (300, 64, 4096, 200),
])
def test_listed_rows_match_oracle(nq, dim, rows, k):
    n = 70_000
    rng = np.random.default_rng(nq + dim)
    x = rng.integers(0, 256, (n, dim)).astype(np.float32)
    cols = np.full((1, n), 5.0)
    cols[0, rng.choice(n, rows, replace=False)] = 1.0
    q = rng.integers(0, 256, (nq, dim)).astype(np.float32)
    bp = pred.concat([Cmp(0, "<", 2.0)] * nq, n)
    gi = GpuIndex(x, cols, device=0, precision=_lib.FV_GPU_PREC_FP32)
    ids, dists, cnt, trunc = gi.brute_batch_raw(q, bp, k)
    assert _lib.lib().pv_last_sparse(gi.handle) == 1
    gi.close()
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q, bp, k)
    for i in range(nq):
        m = int(o_cnt[i])
        assert cnt[i] == m == min(k, rows) and trunc[i] == (rows > k)
        assert np.array_equal(ids[i, :m], o_ids[i, :m].astype(np.uint64))
        assert np.array_equal(dists[i, :m], o_d[i, :m])


@pytest.mark.parametrize("dim", [128, 100, 36])
def test_same_bits_as_the_row_per_warp_kernel(dim):
    # real-valued rows: 12 queries take the tiles, each one alone does not
    n, rows, k = 30_000, 900, 64
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    cols = np.full((1, n), 5.0)
    cols[0, rng.choice(n, rows, replace=False)] = 1.0
    q = rng.standard_normal((12, dim)).astype(np.float32)
    gi = GpuIndex(x, cols, device=0, precision=_lib.FV_GPU_PREC_FP32)
    f = Cmp(0, "<", 2.0)
    ids, dists, cnt, _ = gi.brute_batch(q, [f] * 12, k)
    for s in (slice(0, 9), slice(3, 12)):  # nine queries: gather_dist_kernel
        i2, d2, c2, _ = gi.brute_batch(q[s], [f] * 9, k)
        assert np.array_equal(ids[s], i2) and np.array_equal(cnt[s], c2)
        assert np.array_equal(dists[s].view(np.uint32), d2.view(np.uint32))
    gi.close()
