"""The exact scan of a few queries over the rows their filter passes, against
the oracle: its batch and list limits, word and warp remainders, filters it
tests itself (one range form shared by the batch) and by bitmap (others,
several, some queries without)."""
import numpy as np
import pytest

from oracle import cpu
from paves_b200 import _lib, datagen, pred
from paves_b200.index import GpuIndex
from paves_b200.pred import And, Cmp, In, Not, Or

pytestmark = pytest.mark.gpu
P, C = datagen.COL_PRICE, datagen.COL_CATEGORY
RANGE = And(Cmp(P, ">=", 100.0), Cmp(P, "<", 160.0), In(C, [2, 5, 70]))
FILTERS = {
    "none": lambda n: [None] * n,
    "range": lambda n: [RANGE] * n,
    "narrow": lambda n: [Cmp(P, "==", 3.25)] * n,
    "nothing": lambda n: [Cmp(P, "<", -1.0)] * n,
    "nan": lambda n: [Cmp(P, "<", float("nan"))] * n,
    "tree": lambda n: [Or(RANGE, Not(Cmp(C, "<", 9.0)))] * n,
    "own": lambda n: [None if i % 3 == 2 else Cmp(P, ">", 90.0 * i) for i in range(n)],
}


@pytest.mark.parametrize("n,dim,nq,k", [
    (1, 4, 1, 1), (31, 128, 8, 10), (33, 100, 2, 32), (5000, 128, 1, 64), (20011, 36, 3, 33),
    (20000, 129, 4, 10), (9999, 256, 3, 64), (7000, 512, 2, 10), (7000, 260, 1, 33),
    (40000, 128, 9, 10), (6000, 512, 3, 10), (6000, 128, 5, 65),  # just past its limits
])
@pytest.mark.parametrize("kind", list(FILTERS))
def test_matches_oracle(n, dim, nq, k, kind):
    rng = np.random.default_rng(n + dim)
    x = rng.integers(0, 256, (n, dim)).astype(np.float32)
    cols = np.stack([rng.integers(0, 10, n).astype(np.float64), rng.uniform(0, 1000, n)])
    cols[P, ::5] = np.nan
    cols[P, 3::50] = 3.25
    q = rng.integers(0, 256, (nq, dim)).astype(np.float32)
    preds = FILTERS[kind](nq)
    bp = pred.concat(preds, n)
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q, bp, k)
    for prec in (_lib.FV_GPU_PREC_FP32, _lib.FV_GPU_PREC_BF16):
        gi = GpuIndex(x, cols, device=0, precision=prec)
        ids, dists, cnt, trunc = gi.brute_batch_raw(q, bp, k)
        gi.close()
        for i in range(nq):
            m = int(o_cnt[i])
            assert cnt[i] == m
            assert trunc[i] == (int(pred.eval_numpy(preds[i], cols).sum()) > k)
            assert np.array_equal(ids[i, :m], o_ids[i, :m].astype(np.uint64))
            assert np.array_equal(dists[i, :m], o_d[i, :m])
