"""The exact mode's certificate on rows whose values sit badly with TF32: the
answers are the CUDA-core scan's, whatever share of them it certifies."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["offset", "low bits", "mixed norms", "unit", "huge"])
@pytest.mark.parametrize("dim,topb", [(128, 10), (33, 40)])
def test_answers_are_the_cuda_core_scans(kind, dim, topb):
    rng = np.random.default_rng(len(kind) + dim)
    n, nq = 30_000, 48
    x = rng.standard_normal((n, dim))
    q = rng.standard_normal((nq, dim))
    if kind == "offset":  # truncation pulls every product the same way
        x, q = x + 1000.0, q + 1000.0
    elif kind == "low bits":  # every mantissa bit TF32 drops is set
        x, q = [(a.astype(np.float32).view(np.uint32) | 0x1FFF).view(np.float32) for a in (x, q)]
    elif kind == "mixed norms":
        x *= 10.0 ** rng.uniform(-3, 3, (n, 1))
    elif kind == "unit":
        x /= np.linalg.norm(x, axis=1, keepdims=True)
        q /= np.linalg.norm(q, axis=1, keepdims=True)
    else:
        x *= 1e15
        q *= 1e15
    x, q = x.astype(np.float32), q.astype(np.float32)
    gi = GpuIndex(x, None, device=0)
    ids, dists, cnt, _ = gi.brute_batch(q, [None] * nq, topb)
    assert _lib.lib().pv_last_exact_tc(gi.handle) == 1
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, [None] * nq, topb)
    gi.close()
    assert np.array_equal(cnt, c2)
    # f32 sums in another order: (dim + 8) * 2^-23 of a distance at most
    tol = (dim + 8) * 2.0 ** -23
    np.testing.assert_allclose(dists, d2, rtol=2 * tol)
    for i in range(nq):
        swapped = ids[i] != i2[i]
        for j in np.flatnonzero(swapped):  # rows whose f32 distances tie within it
            assert abs(dists[i, j] - d2[i, j]) <= 2 * tol * d2[i, j]
            true = ((x[int(ids[i, j])].astype(np.float64) - q[i]) ** 2).sum()
            assert abs(true - d2[i, j]) <= 2 * tol * d2[i, j]
