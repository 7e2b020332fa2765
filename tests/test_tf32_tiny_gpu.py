"""Exact batches over rows so small that the squares of what TF32 drops of
them vanish in f32: such rows are not certified by a bound of zero."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,scale", [(16, 1e-21), (16, 1e-22), (16, 1e-20), (64, 1e-21), (160, 3e-22)])
def test_answers_are_the_cuda_core_scans(dim, scale):
    rng = np.random.default_rng(dim)
    n, nq = 20_000, 16  # offsets of fifty spreads: TF32 sees little but the offset
    x = ((50 + rng.standard_normal((n, dim))) * scale).astype(np.float32)
    q = ((50 + rng.standard_normal((nq, dim))) * scale).astype(np.float32)
    gi = GpuIndex(x, None, device=0)
    ids, dists, cnt, _ = gi.brute_batch(q, [None] * nq, 10)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, [None] * nq, 10)
    gi.close()
    assert np.array_equal(cnt, c2) and np.array_equal(ids, i2) and np.array_equal(dists, d2)
