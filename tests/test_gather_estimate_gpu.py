"""The estimated bound of large supersets on gathered sets that have room for
more rows than pass (a filter of two terms, bounded by the closer one): no
query falls short of its superset, so none is run twice."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import And, Cmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,nq,k,a,b,prec,gathered", [
    (1_000_000, 96, 256, 75, 0.2, 0.5, _lib.FV_GPU_PREC_FP8, 1),
    (600_001, 64, 129, 55, 0.2, 0.3, _lib.FV_GPU_PREC_FP8, 0),
    (600_001, 128, 300, 120, 0.3, 0.5, _lib.FV_GPU_PREC_FP8, 1),
    (400_003, 96, 512, 90, 0.35, 0.7, _lib.FV_GPU_PREC_FP8, 1),
    (1_000_000, 128, 200, 100, 0.15, 0.5, _lib.FV_GPU_PREC_BF16, 1),
    (500_000, 128, 257, 70, 0.3, 0.2, _lib.FV_GPU_PREC_BF16, 1),
    (600_001, 96, 300, 75, 0.2, 1.0, _lib.FV_GPU_PREC_FP8, 1),
    (600_001, 96, 300, 75, 0.25, 0.93, _lib.FV_GPU_PREC_FP8, 1),
])
def test_nothing_is_run_twice(n, dim, nq, k, a, b, prec, gathered):
    rng = np.random.default_rng(n + nq + k)
    x = rng.integers(0, 128, (n, dim)).astype(np.float32)
    q = rng.integers(0, 128, (nq, dim)).astype(np.float32)
    cols = rng.uniform(0, 1, (2, n))
    f = And(Cmp(0, "<", a), Cmp(1, "<", b))
    gi = GpuIndex(x, cols, device=0, precision=prec)
    ids, dists, cnt, _ = gi.brute_batch(q, [f] * nq, k)
    L = _lib.lib()
    unc, S = L.pv_last_uncertain(gi.handle), L.pv_last_superset(gi.handle)
    sparse = L.pv_last_sparse(gi.handle)
    gi.close()
    assert S > 64 and unc == 0
    assert sparse == gathered
    assert (cnt == k).all()
    rows = np.flatnonzero((cols[0] < a) & (cols[1] < b))
    if prec == _lib.FV_GPU_PREC_BF16:  # exact distances: the oracle on a few queries
        for i in range(0, nq, 37):
            d = ((x[rows] - q[i]) ** 2).sum(1)
            want = rows[np.lexsort((rows, d))[:k]]
            assert np.array_equal(ids[i], want)
