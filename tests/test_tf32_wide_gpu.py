"""Rows beyond 128 dims on the tensor cores (the query tile streams with the
rows): the CUDA-core scans' answers bit for bit, on FP32 uploads and on BF16
uploads too wide for their own scan; whole and ragged K-blocks."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu
LOW = _lib.FV_GPU_PREC_BF16


@pytest.mark.parametrize("dim,nq,k,prec", [
    (129, 16, 10, 0), (160, 33, 1, 0), (200, 24, 64, 0), (200, 23, 64, 0), (256, 64, 10, 0),
    (256, 130, 65, 0), (260, 16, 10, LOW), (384, 33, 50, 0), (384, 65, 10, LOW), (500, 200, 10, 0),
    (512, 128, 250, 0), (512, 20, 3, LOW),
])
@pytest.mark.parametrize("share", [1.0, 0.4])
def test_same_as_the_cuda_core_scan(dim, nq, k, prec, share):
    rng = np.random.default_rng(dim + nq)
    n = 9001 if dim > 300 else 20_003
    centers = rng.uniform(0, 128, (16, dim))
    x = (centers[rng.integers(0, 16, n)] + rng.normal(0, 20, (n, dim))).astype(np.float32)
    q = (centers[rng.integers(0, 16, nq)] + rng.normal(0, 20, (nq, dim))).astype(np.float32)
    cols = rng.uniform(0, 1, (1, n))
    preds = [Cmp(0, "<", share)] * (nq - 1) + [Cmp(0, "<", 0.9)]
    gi = GpuIndex(x, cols, device=0, precision=prec)
    ids, dists, cnt, trunc = gi.brute_batch(q, preds, k)
    assert _lib.lib().pv_last_exact_tc(gi.handle) == 1
    unc = _lib.lib().pv_last_uncertain(gi.handle)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, t2 = gi.brute_batch(q, preds, k)
    gi.close()
    assert unc < nq
    assert np.array_equal(cnt, c2) and np.array_equal(trunc, t2)
    if unc == 0:  # (re-run queries take the order of a smaller batch)
        assert np.array_equal(dists.view(np.uint32), d2.view(np.uint32))
        assert np.array_equal(ids, i2)
    np.testing.assert_allclose(dists, d2, rtol=2e-6)


def test_selective_filter_on_wide_rows():
    rng = np.random.default_rng(8)
    n, dim, nq, k = 400_000, 192, 40, 10
    x = rng.standard_normal((n, dim), dtype=np.float32)
    cols = rng.uniform(0, 1, (1, n))
    q = rng.standard_normal((nq, dim), dtype=np.float32)
    preds = [Cmp(0, "<", 0.05)] * nq  # 20,000 rows: the compacted set
    gi = GpuIndex(x, cols, device=0)
    ids, dists, cnt, _ = gi.brute_batch(q, preds, k)
    assert _lib.lib().pv_last_sparse(gi.handle) == 1 == _lib.lib().pv_last_exact_tc(gi.handle)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, preds, k)
    gi.close()
    assert np.array_equal(cnt, c2) and np.array_equal(ids, i2)
    assert np.array_equal(dists.view(np.uint32), d2.view(np.uint32))
