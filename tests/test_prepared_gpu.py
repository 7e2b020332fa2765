"""Prepared batches report uncertified queries and do not re-run them, so
what was exact without a certificate stays so: rows beyond 128 dims, and
supersets that whole lists hold."""
import ctypes as C

import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib, pred
from paves_b200._lib import HIT_DTYPE, ptr

pytestmark = pytest.mark.gpu


def prepared(gi, q, preds, k, mode):
    L = _lib.lib()
    bp = pred.concat(preds, gi.count)
    err = C.create_string_buffer(256)
    nq = len(q)
    b = L.pv_batch_create(gi.handle, nq, ptr(q), ptr(bp.qd), ptr(bp.nodes), len(bp.nodes),
                          ptr(bp.children), len(bp.children), ptr(bp.invals), len(bp.invals), k,
                          mode, err, 256)
    assert b, err.value
    out, cnt = np.zeros(nq * k, HIT_DTYPE), np.zeros(nq, np.uint32)
    tr = np.zeros(nq, np.uint8)
    assert L.pv_batch_run(b, 2, None, None, err, 256) == 0, err.value
    assert L.pv_batch_fetch(b, ptr(out), ptr(cnt), ptr(tr), err, 256) == 0, err.value
    L.pv_batch_free(b)
    out = out.reshape(nq, k)
    return out["node"], out["dist"], cnt, tr, L.pv_last_uncertain(gi.handle)


@pytest.mark.parametrize("dim,prec,mode", [(200, 0, _lib.PV_MODE_EXACT), (512, 0, _lib.PV_MODE_EXACT),
                                           (300, _lib.FV_GPU_PREC_BF16, _lib.PV_MODE_LOW)])
def test_wide_rows(dim, prec, mode):
    rng = np.random.default_rng(dim)
    n, nq, k = 12_000, 33, 10  # an offset at which TF32 certifies few queries or none
    x = (40 + rng.standard_normal((n, dim))).astype(np.float32)
    q = (40 + rng.standard_normal((nq, dim))).astype(np.float32)
    gi = GpuIndex(x, None, device=0, precision=prec)
    ids, dists, cnt, _, unc = prepared(gi, q, [None] * nq, k, mode)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    i2, d2, c2, _ = gi.brute_batch(q, [None] * nq, k)
    gi.close()
    assert unc == 0
    assert np.array_equal(cnt, c2) and np.array_equal(ids, i2) and np.array_equal(dists, d2)


@pytest.mark.parametrize("block", [4000, 9000])
def test_whole_lists(block):
    """More rows within every query's bound than the short lists' runs hold
    (a cluster of consecutive rows in a table that is otherwise mixed)."""
    rng = np.random.default_rng(block)
    n, dim, nq, k = 150_000, 64, 1024, 64
    x = rng.integers(0, 200, (n, dim)).astype(np.float32)
    x[30_000:30_000 + block] = 100 + rng.integers(-3, 4, (block, dim))
    q = (100 + rng.integers(-3, 4, (nq, dim))).astype(np.float32)
    gi = GpuIndex(x, None, device=0, precision=_lib.FV_GPU_PREC_BF16)
    ids, dists, cnt, _, unc = prepared(gi, q, [None] * nq, k, _lib.PV_MODE_LOW)
    gi.close()
    ex = GpuIndex(x, None, device=0)
    assert _lib.lib().pv_exact_tc(ex.handle, 0) == 0
    i2, d2, c2, _ = ex.brute_batch(q, [None] * nq, k)
    ex.close()
    assert unc == 0
    assert np.array_equal(cnt, c2) and np.array_equal(ids, i2) and np.array_equal(dists, d2)
