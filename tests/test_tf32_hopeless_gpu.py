"""Wide rows whose offset hides their differences from TF32 stay on the
CUDA-core scan (every query would be scanned twice); rows that TF32 tells
apart take the tensor cores."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [132, 200, 512])
@pytest.mark.parametrize("offset,tc", [(0.0, 1), (1000.0, 0)])
@pytest.mark.parametrize("clusters", [1, 300])
def test_route(dim, offset, tc, clusters):
    rng = np.random.default_rng(dim)
    n, nq = 12_000, 33
    c = rng.normal(0, 6, (clusters, dim)) * (clusters > 1)
    x = (c[rng.integers(0, clusters, n)] + rng.standard_normal((n, dim)) + offset).astype(np.float32)
    q = (c[rng.integers(0, clusters, nq)] + rng.standard_normal((nq, dim)) + offset).astype(np.float32)
    gi = GpuIndex(x, None, device=0)
    ids, dists, cnt, _ = gi.brute_batch(q, [None] * nq, 10)
    took = _lib.lib().pv_last_exact_tc(gi.handle)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, [None] * nq, 10)
    gi.close()
    assert took == tc
    assert np.array_equal(cnt, c2) and np.array_equal(ids, i2)
    np.testing.assert_allclose(dists, d2, rtol=2 * (dim + 8) * 2.0 ** -23)
