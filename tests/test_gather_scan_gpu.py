"""A filter shared by the whole batch that passes some percent of a large
table: its rows are gathered and scanned. The answers are those of the scan
over the whole index (the same filter as two programs), bit for bit."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import And, Cmp

pytestmark = pytest.mark.gpu
F32, BF16, FP8 = 0, _lib.FV_GPU_PREC_BF16, _lib.FV_GPU_PREC_FP8


@pytest.mark.parametrize("prec,n,nq,k,share,real,gathered", [
    (BF16, 600_001, 1, 10, 0.07, False, 1), (BF16, 600_001, 33, 1, 0.1, True, 1),
    (BF16, 600_001, 130, 64, 0.15, False, 1), (BF16, 600_001, 130, 64, 0.25, False, 0),
    (BF16, 600_001, 300, 10, 0.4, True, 1), (F32, 400_033, 24, 10, 0.1, False, 1),
    (F32, 400_033, 64, 50, 0.15, True, 1), (F32, 400_033, 257, 128, 0.35, False, 1),
    (FP8, 600_001, 16, 10, 0.1, False, 1), (FP8, 600_001, 129, 25, 0.15, True, 1),
    (FP8, 600_001, 129, 25, 0.2, True, 0),
])
@pytest.mark.parametrize("loose", [False, True])
def test_same_as_the_scan_of_the_index(prec, n, nq, k, share, real, gathered, loose):
    rng = np.random.default_rng(n + nq + k)
    x = rng.integers(0, 128, (n, 128)).astype(np.float32)
    q = rng.integers(0, 128, (nq, 128)).astype(np.float32)
    if real:
        x += rng.standard_normal((n, 128), dtype=np.float32)
        q += rng.standard_normal((nq, 128), dtype=np.float32)
    cols = rng.uniform(0, 1, (2, n))

    def one(a):  # loose: the bound on the passing rows is twice their number
        return And(Cmp(0, "<", a), Cmp(1, "<", 0.5)) if loose else Cmp(0, "<", a)

    gi = GpuIndex(x, cols, device=0, precision=prec)
    ids, dists, cnt, trunc = gi.brute_batch(q, [one(share)] * nq, k)
    assert _lib.lib().pv_last_sparse(gi.handle) == gathered
    unc = _lib.lib().pv_last_uncertain(gi.handle)
    # the same rows from a second program, one query of padding
    two = [one(share)] * nq + [one(0.9)]
    i2, d2, c2, t2 = gi.brute_batch(np.vstack([q, q[:1]]), two, k)
    assert _lib.lib().pv_last_sparse(gi.handle) == 0
    gi.close()
    assert unc <= nq // 8
    assert np.array_equal(cnt, c2[:nq]) and np.array_equal(trunc, t2[:nq])
    assert np.array_equal(ids, i2[:nq])
    assert np.array_equal(dists.view(np.uint32), d2[:nq].view(np.uint32))
