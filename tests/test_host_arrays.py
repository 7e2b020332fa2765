"""The batch's predicate arrays and the integer-row certificate, on the host."""
import numpy as np
import pytest

from paves_b200 import _lib, pred
from paves_b200.pred import And, Cmp, In, Not, Or


def test_concat_places_every_querys_own_slice():
    trees = [And(Cmp(0, "<", 3.0), In(1, [1, 2, 5])), None, Not(Or(Cmp(1, "==", 2), And(), In(0, []))),
             Cmp(0, "!=", float("nan"))]
    order = [0, 2, 0, 1, 3, 2, 0]
    bp = pred.concat([trees[i] for i in order], 77, entries=list(range(7)))
    n = c = v = 0
    for q, i in enumerate(order):
        if trees[i] is None:
            assert bp.qd[q]["proot"] == bp.roots[q] == -1
            continue
        s = pred.serialize(trees[i])
        assert bp.qd[q]["proot"] == bp.roots[q] == n
        want = s.nodes.copy()
        want["child0"] += c
        want["val0"] += v
        assert bp.nodes[n:n + len(want)].tobytes() == want.tobytes()
        assert np.array_equal(bp.children[c:c + len(s.children)], s.children + n)
        assert np.array_equal(bp.invals[v:v + len(s.invals)], s.invals)
        n, c, v = n + len(want), c + len(s.children), v + len(s.invals)
    assert (len(bp.nodes), len(bp.children), len(bp.invals)) == (n, c, v)
    assert list(bp.qd["entry"]) == list(range(7)) and (bp.qd["total"] == 77).all()


@pytest.mark.parametrize("entries", [[3], [1, 2], np.array([4]), [-1, 0, 0]])
def test_entries_that_are_refused(entries):
    with pytest.raises((IndexError, OverflowError)):
        pred.concat([None] * 3, 10, entries=entries)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4095, 4096, 4105])
@pytest.mark.parametrize("odd", [None, 0.5, 257.0, -257.0, np.nan, np.inf, -np.inf, 1e-40])
def test_integral_amax(n, odd):
    x = np.random.default_rng(n).integers(-256, 257, n).astype(np.float32)
    for at in {0, n // 2, n - 1}:
        y = x.copy()
        if odd is not None:
            y[at] = odd
        want = float(np.abs(x).max()) if odd is None else -1.0
        assert _lib.lib().pv_rows_integral_amax(_lib.ptr(y), n) == want
