"""Batches of several range-form filters (the position-form bitmaps) against
the oracle: program counts around the 32-program chunks, rows around the warps' shares,
NaN / infinite / tied values, and posting rows that are no ordering."""
import numpy as np
import pytest

from oracle import cpu
from paves_b200 import datagen, pred
from paves_b200.index import GpuIndex
from paves_b200.pred import And, Cmp, In

pytestmark = pytest.mark.gpu
P, C = datagen.COL_PRICE, datagen.COL_CATEGORY


def table(n, seed, top):
    rng = np.random.default_rng(seed)
    cols = np.stack([rng.integers(0, top, n).astype(np.float64),
                     np.round(rng.uniform(-50, 1000, n)), rng.uniform(0, 1, n)])
    cols[1, ::7] = np.nan
    cols[1, 3::11] = np.inf
    cols[1, 5::13] = -np.inf
    cols[1, 1::17] = -0.0
    cols[0, 2::19] = np.nan
    cols[2, 4::5] = 31.0
    return rng.integers(0, 256, (n, 32)).astype(np.float32), cols


def filters(rng, m, top):
    out = []
    for i in range(m):
        a = float(rng.uniform(-60, 900))
        f = [Cmp(P, ">=", a) & Cmp(P, "<", a + float(rng.uniform(0, 400))),
             Cmp(P, "==", float(rng.integers(-1, 3))), Cmp(P, ">", np.inf), Cmp(P, ">=", np.inf),
             Cmp(P, "<=", -np.inf), Cmp(P, "<", np.nan), Cmp(2, "<", float(rng.uniform(0, 1))),
             Cmp(C, ">", 1.0) & Cmp(P, "<=", a)][int(rng.integers(8))]
        if rng.random() < 0.5:
            f = And(f, In(C, [float(v) for v in rng.integers(0, top + 3, 4)]))
        if rng.random() < 0.2:
            f = In(C, [float(rng.integers(0, top))])
        out.append(f)
    return out


@pytest.mark.parametrize("n,m,top,order", [
    (1500, 8, 10, "kept"), (1024, 9, 31, "kept"), (3333, 32, 10, "kept"), (2049, 33, 31, "kept"),
    (31, 12, 10, "kept"), (70001, 300, 10, "kept"), (8192, 1024, 31, "kept"),
    (2049, 33, 40, "kept"),      # integers a code byte cannot hold: the f64 columns
    (2049, 33, 10, "reversed"),  # posting rows in no order
    (2049, 33, 10, "repeated"),  # a row listed twice
])
def test_many_filters_match_oracle(n, m, top, order):
    x, cols = table(n, n + m, top)
    rng = np.random.default_rng(m)
    preds = filters(rng, m, top)
    q = rng.integers(0, 256, (m, 32)).astype(np.float32)
    post = datagen.posting_rows(cols)
    if order == "reversed":
        post = post[:, ::-1].copy()
    if order == "repeated":
        post[:, 5] = post[:, 6]
    gi = GpuIndex(x, cols, post_rows=post, device=0)
    bp = pred.concat(preds, n)
    ids, dists, cnt, trunc = gi.brute_batch_raw(q, bp, 8)
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q, bp, 8)
    for i in range(m):
        passing = int(pred.eval_numpy(preds[i], cols).sum())
        assert cnt[i] == o_cnt[i] == min(8, passing)
        assert trunc[i] == (passing > 8)
        assert np.array_equal(ids[i, :cnt[i]], o_ids[i, :cnt[i]].astype(np.uint64))
        assert np.array_equal(dists[i, :cnt[i]], o_d[i, :cnt[i]])
    gi.close()
