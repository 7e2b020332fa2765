"""Whose summation order the exact mode's answers carry: the CUDA-core scan's
wherever that scan gave the answer before a closer bound or a wider kernel
took over."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu


def both_routes(x, cols, q, preds, k):
    gi = GpuIndex(x, cols, device=0)
    got = gi.brute_batch(q, preds, k)
    took = _lib.lib().pv_last_exact_tc(gi.handle), _lib.lib().pv_last_sparse(gi.handle)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    want = gi.brute_batch(q, preds, k)
    gi.close()
    return got, want, took


def same(got, want):
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("dim,nq,k", [(128, 16, 10), (128, 23, 40), (64, 20, 10), (36, 16, 5)])
def test_rows_that_only_the_closer_bound_separates(dim, nq, k):
    """An offset at which the bound that any values allow (2^-8 ||x|| ||q||)
    is larger than the distances' gaps, and the rows' own residual is not."""
    rng = np.random.default_rng(dim)
    n = 20_000
    x = (7 + rng.standard_normal((n, dim))).astype(np.float32)
    q = (7 + rng.standard_normal((nq, dim))).astype(np.float32)
    got, want, (tc, _) = both_routes(x, None, q, [None] * nq, k)
    assert tc == 1
    same(got, want)


@pytest.mark.parametrize("dim,nq,k,n", [(200, 32, 10, 400_000), (256, 24, 64, 300_000),
                                        (160, 100, 1, 500_000), (200, 23, 10, 600_000),
                                        (300, 130, 10, 200_000), (200, 64, 80, 300_000)])
def test_gathered_wide_rows(dim, nq, k, n):
    """A shared filter of 10 % is scanned as a gathered set; the sums are
    those of the scan of the index."""
    rng = np.random.default_rng(dim + nq)
    x = rng.standard_normal((n, dim), dtype=np.float32)
    q = rng.standard_normal((nq, dim), dtype=np.float32)
    cols = rng.uniform(0, 1, (1, n))
    got, want, took = both_routes(x, cols, q, [Cmp(0, "<", 0.1)] * nq, k)
    assert took == (1, 1)
    same(got, want)
