"""Batches of two to eight range-form filters (bitmap_few_kernel) against the
oracle: rows around a warp's and a block's share, one and several terms a
filter, columns in and beyond the general kernel's registers, NaN, infinite
and signed-zero values."""
import numpy as np
import pytest

from oracle import cpu
from paves_b200 import datagen, pred
from paves_b200.index import GpuIndex
from paves_b200.pred import And, Cmp, In

pytestmark = pytest.mark.gpu


def table(n, ncols):
    rng = np.random.default_rng(n + ncols)
    cols = np.round(rng.uniform(-5, 70, (ncols, n)))
    cols[1:, 1::2] += 0.5
    cols[0, ::7] = np.nan
    cols[ncols - 1, 3::11] = np.inf
    cols[0, 5::13] = -np.inf
    cols[0, 1::17] = -0.0
    return rng.integers(0, 256, (n, 32)).astype(np.float32), cols


@pytest.mark.parametrize("n", [1, 31, 127, 129, 2047, 2048, 2049, 70001])
@pytest.mark.parametrize("ncols,m", [(1, 2), (2, 8), (3, 5), (6, 8)])
def test_few_filters_match_oracle(n, ncols, m):
    x, cols = table(n, ncols)
    rng = np.random.default_rng(m)
    preds = []
    for i in range(m):
        terms = []
        for c in sorted(rng.choice(ncols, min(ncols, 1 + i % 4), replace=False).tolist()):
            lo = float(rng.integers(-6, 40))
            terms.append([And(Cmp(c, ">=", lo), Cmp(c, "<", lo + 45)), Cmp(c, "<=", lo + 40),
                          In(c, [float(v) for v in rng.integers(0, 64, 30)]), Cmp(c, ">", lo - 30),
                          And(In(c, [0.0, 1.0, 63.0]), Cmp(c, ">=", 0.0))][int(rng.integers(5))])
        preds.append(terms[0] if len(terms) == 1 else And(*terms))
    nq = 3 * m
    preds = [preds[i % m] for i in range(nq)]
    q = rng.integers(0, 256, (nq, 32)).astype(np.float32)
    gi = GpuIndex(x, cols, post_rows=datagen.posting_rows(cols), device=0)
    bp = pred.concat(preds, n)
    ids, dists, cnt, trunc = gi.brute_batch_raw(q, bp, 8)
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q, bp, 8)
    for i in range(nq):
        passing = int(pred.eval_numpy(preds[i], cols).sum())
        assert cnt[i] == o_cnt[i] == min(8, passing)
        assert trunc[i] == (passing > 8)
        assert np.array_equal(ids[i, :cnt[i]], o_ids[i, :cnt[i]].astype(np.uint64))
        assert np.array_equal(dists[i, :cnt[i]], o_d[i, :cnt[i]])
    gi.close()
