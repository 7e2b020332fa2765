"""Predicate arrays: every query's slice on both ways they are written (in
place up to eight filters, gathered beyond), and what is refused or taken."""
import numpy as np
import pytest

from paves_b200 import pred
from paves_b200.pred import And, Cmp, In, Not, Or

TREES = [And(Cmp(0, "<", 3.0), In(1, [1, 2, 5])), None,
         Not(Or(Cmp(1, "==", 2), And(), In(0, []))), Cmp(0, "!=", float("nan"))]


@pytest.mark.parametrize("order", [
    [0, 2, 0, 1, 3, 2, 0], [0, 2, 0, 1, 3, 2, 0] * 3, [0, 3, 2, 2, 0, 1, 1, 3, 3, 2],
    [0, 3, 2, 2, 0, 1, 1, 3, 3, 2, 0], [1] * 12, [2] * 9, [1, 3] * 10, [],
])
def test_every_querys_own_slice(order):
    bp = pred.concat([TREES[i] for i in order], 77, entries=list(range(len(order))))
    n = c = v = 0
    for q, i in enumerate(order):
        if TREES[i] is None:
            assert bp.qd[q]["proot"] == bp.roots[q] == -1
            continue
        s = pred.serialize(TREES[i])
        assert bp.qd[q]["proot"] == bp.roots[q] == n
        want = s.nodes.copy()
        want["child0"] += c
        want["val0"] += v
        assert bp.nodes[n:n + len(want)].tobytes() == want.tobytes()
        assert np.array_equal(bp.children[c:c + len(s.children)], s.children + n)
        assert np.array_equal(bp.invals[v:v + len(s.invals)], s.invals)
        n, c, v = n + len(want), c + len(s.children), v + len(s.invals)
    assert (len(bp.nodes), len(bp.children), len(bp.invals)) == (n, c, v)
    assert (bp.nodes.dtype, bp.children.dtype, bp.invals.dtype) == (
        pred.NODE_DTYPE, np.int32, np.float64)
    assert list(bp.qd["entry"]) == list(range(len(order))) and (bp.qd["total"] == 77).all()


@pytest.mark.parametrize("col,error", [(2 ** 31, OverflowError), (-2 ** 31 - 1, OverflowError),
                                       (2 ** 40, OverflowError), (np.uint64(2 ** 40), OverflowError),
                                       (None, TypeError), ("x", ValueError)])
@pytest.mark.parametrize("queries", [1, 9])
def test_columns_that_are_refused(col, error, queries):
    for p in (Cmp(col, "<", 1.0), In(col, [1.0])):
        with pytest.raises(error):
            pred.concat([p] * queries, 10)


@pytest.mark.parametrize("col", [1, np.int64(1), np.uint8(1), True, np.float32(1.5), "1", np.array(1)])
def test_columns_that_are_taken(col):
    for p in (Cmp(col, "<", 1.0), In(col, [1.0])):
        assert pred.serialize(p).nodes["col"][0] == 1


@pytest.mark.parametrize("queries", [1, 9])
@pytest.mark.parametrize("thing", [3, "s", And])
def test_what_is_no_predicate(thing, queries):
    for p in (thing, And(Cmp(0, "<", 1.0), thing)):
        with pytest.raises(KeyError):
            pred.concat([p] * queries, 10)


@pytest.mark.parametrize("entries", [[3, 4, 5], (3, 4, 5, 6), range(3, 6), {0: 3, 1: 4, 2: 5},
                                     np.array([3, 4, 5]), np.float32([3, 4, 5]),
                                     np.array([3, 4, 5], object), "345"])
def test_entries_that_are_taken(entries):
    assert pred.concat([None] * 3, 10, entries=entries).qd["entry"].tolist() == [3, 4, 5]
