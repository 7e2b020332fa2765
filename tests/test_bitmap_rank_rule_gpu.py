"""Batches of many range-form filters on tables large enough for the
position-form bitmaps, and one row or filter short of that, against the
oracle: program counts around the 32-program chunks, rows around the words
and shares of a warp."""
import numpy as np
import pytest

from oracle import cpu
from paves_b200 import _lib, datagen, pred
from paves_b200.index import GpuIndex
from paves_b200.stream import Stream
from tests.test_bitmap_rank_gpu import filters, table

pytestmark = pytest.mark.gpu


def rows_from(m):
    """The smallest table on which m programs take the position form."""
    return -(-(2_400_000 + 25_000 * m) // m)


@pytest.mark.parametrize("m,more", [(9, 0), (9, -1), (32, 17), (33, 1), (64, 0), (300, 255), (513, 0),
                                    (1024, -1), (1024, 0), (1024, 31)])
@pytest.mark.parametrize("top", [10, 31])
def test_many_filters_match_oracle(m, more, top):
    n = rows_from(m) + more
    x, cols = table(n, m + top, top)
    rng = np.random.default_rng(m)
    preds = filters(rng, m, top)
    q = rng.integers(0, 256, (m, 32)).astype(np.float32)
    gi = GpuIndex(x, cols, post_rows=datagen.posting_rows(cols), device=0)
    check(gi, x, cols, q, preds)
    gi.close()


def check(gi, x, cols, q, preds, k=8, run=None):
    bp = pred.concat(preds, len(x))
    if run:
        ids, dists, cnt, _ = run(q, preds, k)
        trunc = None
    else:
        ids, dists, cnt, trunc = gi.brute_batch_raw(q, bp, k)
    some = np.arange(0, len(q), max(1, len(q) // 64))
    bs = pred.concat([preds[i] for i in some], len(x))
    o_ids, _, o_d, o_cnt, _ = cpu.exact_topk(x, cols, q[some], bs, k)
    for i in range(len(q)):
        passing = int(pred.eval_numpy(preds[i], cols).sum())
        assert cnt[i] == min(k, passing)
        assert trunc is None or trunc[i] == (passing > k)
    for j, i in enumerate(some):
        assert np.array_equal(ids[i, :cnt[i]], o_ids[j, :cnt[i]].astype(np.uint64))
        assert np.array_equal(dists[i, :cnt[i]], o_d[j, :cnt[i]])


@pytest.mark.parametrize("n", [60_000, 120_000])
def test_streams_choose_by_batch(n):
    """One graph serves batches of either form: 64 selective filters take the
    position form on the larger table only, 12 on neither."""
    x, cols = table(n, 3, 10)
    rng = np.random.default_rng(5)
    gi = GpuIndex(x, cols, post_rows=datagen.posting_rows(cols), device=0,
                  precision=_lib.FV_GPU_PREC_BF16)
    q = rng.integers(0, 256, (64, 32)).astype(np.float32)
    s = Stream(gi, 64, 8, q)
    for m in (64, 12, 40, 64, 3):
        check(gi, x, cols, q[:m], filters(rng, m, 10), run=s.run)
    s.close()
    gi.close()
