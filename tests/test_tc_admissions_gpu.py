"""Lanes of a warp that part over the rows they admit (a filter of its own
per query, lists that fill, become heaps or spill, with and without a seeded
bound) meet again at every read of the accumulators: the exact answers, for
each number of epilogue groups and operand kind."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu
BF16, FP8 = _lib.FV_GPU_PREC_BF16, _lib.FV_GPU_PREC_FP8


@pytest.mark.parametrize("prec", [0, BF16, FP8])
@pytest.mark.parametrize("epi,nq,k", [(1, 128, 64), (2, 40, 10), (2, 128, 64), (3, 128, 60), (3, 300, 7)])
@pytest.mark.parametrize("seed", [0, 2])
def test_lanes_part_and_meet(prec, epi, nq, k, seed):
    rng = np.random.default_rng(nq + k)
    n, dim = 30_001, 96
    x = rng.integers(0, 100, (n, dim)).astype(np.float32)
    q = rng.integers(0, 100, (nq, dim)).astype(np.float32)
    cols = rng.uniform(0, 1, (1, n))
    share = np.where(np.arange(nq) % 3 == 0, 0.9, 0.02 + rng.uniform(0, 0.5, nq))
    preds = [Cmp(0, "<", float(s)) for s in share]
    gi = GpuIndex(x, cols, device=0, precision=prec)
    L = _lib.lib()
    assert L.pv_tc_shape(gi.handle, epi, 2, 0, 0, seed) == 0
    ids, dists, cnt, _ = gi.brute_batch(q, preds, k)
    gi.close()
    assert (cnt == k).all()
    hits = 0
    for i in range(nq):
        rows = np.flatnonzero(cols[0] < share[i])
        d = ((x[rows] - q[i]) ** 2).sum(1, dtype=np.float32)
        want = rows[np.lexsort((rows, d))[:k]]
        hits += np.isin(want, ids[i].astype(np.int64)).sum()
        if prec != FP8:
            assert np.array_equal(ids[i], want) and np.array_equal(dists[i], np.sort(d)[:k])
    assert hits >= 0.95 * nq * k  # FP8: approximate by contract
