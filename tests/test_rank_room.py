"""The optional arrays for batches of many filters yield to what calls need."""
import pytest

from paves_b200 import _lib

GB = 1 << 30
TOTAL = 180 * GB


@pytest.mark.parametrize("count,ncols", [(1, 1), (1_000_000, 2), (10_000_000, 4), (400_000_000, 1),
                                         (4_000_000_000, 3)])
def test_room_for_calls_and_a_quarter(count, ncols):
    fit = _lib.lib().pv_rank_tables_fit
    tables = 13 * count * ncols
    # bitmaps and visited sets of 1024 queries, and scratch of up to 1 GB twice
    calls = 2 * 1024 * ((count + 31) // 32) * 4 + 2 * GB
    need = tables + max(calls, TOTAL // 4)
    assert fit(need + 4096, TOTAL, count, ncols) == 1
    assert fit(need - 1, TOTAL, count, ncols) == 0
    assert fit(tables, TOTAL, count, ncols) == fit(0, TOTAL, count, ncols) == 0
    assert fit(1 << 62, TOTAL, count, 0) == fit(1 << 62, TOTAL, count, 5) == 0
