"""Batches of several selective filters over small tables are not seeded (their
lists fill little), broad ones are; the answers are the oracle's."""
import numpy as np
import pytest

from oracle import cpu
from paves_b200 import GpuIndex, _lib, pred
from paves_b200.pred import Cmp, Not, Or

pytestmark = pytest.mark.gpu
BF16, FP8 = _lib.FV_GPU_PREC_BF16, _lib.FV_GPU_PREC_FP8


def each(share, i):
    return Cmp(0, "<", share * (1 + i / 64))


def two(share, i):  # no range form: bounded by the columns' counts
    return Or(Cmp(0, "<", share / 2), Not(Cmp(0, "<", 1 - share / 2))) if i % 2 else Cmp(0, "<", share)


@pytest.mark.parametrize("n,dim,nq,k,prec,form,share,seeded", [
    (8_650, 128, 6, 9, BF16, each, 0.0015, 0), (8_650, 128, 64, 9, BF16, each, 0.9, 1),
    (20_000, 96, 3, 2, FP8, each, 0.01, 0), (60_000, 32, 16, 3, BF16, two, 0.001, 0),
    (40_000, 32, 38, 27, 0, each, 0.01, 0), (40_000, 32, 38, 27, 0, two, 0.8, 1),
    (120_000, 64, 40, 30, BF16, two, 0.5, 1),
])
def test_seeding(n, dim, nq, k, prec, form, share, seeded):
    rng = np.random.default_rng(n + nq)
    x = rng.integers(0, 100, (n, dim)).astype(np.float32)
    q = rng.integers(0, 100, (nq, dim)).astype(np.float32)
    cols = rng.uniform(0, 1, (1, n))
    preds = [form(share, i) for i in range(nq)]
    bp = pred.concat(preds, n)
    gi = GpuIndex(x, cols, device=0, precision=prec)
    L = _lib.lib()
    ids, dists, cnt, _ = gi.brute_batch_raw(q, bp, k)
    launches = L.pv_last_launches(gi.handle)
    assert L.pv_tc_shape(gi.handle, 0, 0, 0, 0, 2) == 0  # never seeded
    i2, d2, c2, _ = gi.brute_batch_raw(q, bp, k)
    assert launches - L.pv_last_launches(gi.handle) == 2 * seeded
    gi.close()
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q, bp, k)
    assert np.array_equal(cnt, o_cnt) and np.array_equal(c2, o_cnt)
    if prec != FP8:
        for i in range(nq):
            c = int(cnt[i])
            assert np.array_equal(ids[i, :c], o_ids[i, :c].astype(np.uint64))
            assert np.array_equal(dists[i, :c], o_d[i, :c])
            assert np.array_equal(i2[i, :c], ids[i, :c])
