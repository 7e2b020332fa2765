"""The graph search's two-part frontier against a plain restatement of the
search (sorted lists on the host): merges of the recent entries into the
rest, the 8192-entry limit, drained frontiers, visit limits, beam widths."""
import numpy as np
import pytest

from paves_b200.index import GpuIndex
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu
FRONTIER, WMAX = 8192, 16


def search(x, lists, q, entry, mask, ef, max_visited, width):
    def dist(i):
        return ((x[i] - q) ** 2).sum()

    seen = {entry}
    front = [(dist(entry), entry)]
    res = [front[0]] if mask[entry] else []
    dropped = False
    while True:
        if not front:
            return res, not dropped
        if len(seen) >= max_visited:
            return res, True
        worst = res[ef - 1][0] if len(res) >= ef else np.inf
        if front[0][0] > worst:
            return res, False
        take = front[:width]
        take = take[:1] + [t for t in take[1:] if t[0] <= worst]
        front = front[len(take):]
        new = []
        for _, v in take:
            for u in lists[v]:
                if u not in seen:
                    seen.add(u)
                    new.append(u)
        new = [(dist(u), u) for u in new]
        new = sorted(n for n in new if len(res) < ef or n[0] < worst)
        res = sorted(res + [n for n in new if mask[n[1]]])[:ef]
        front = sorted(front + new)
        before = len(front)
        if len(res) >= ef:
            front = [f for f in front if f[0] <= res[ef - 1][0]]
        front = front[:FRONTIER]
        dropped = dropped or len(front) < before


@pytest.mark.parametrize("n,deg,ef,share,max_visited", [
    (3000, 32, 40, 0.02, 200000),     # merges of the recent entries, drained
    (30000, 32, 30, 0.0005, 200000),  # more than the frontier holds
    (30000, 32, 200, 0.003, 9000),    # visit limit
    (4000, 7, 512, 0.5, 200000), (4000, 60, 16, 1.0, 200000), (500, 32, 64, 0.0, 200000),
])
def test_matches_plain_search(n, deg, ef, share, max_visited):
    rng = np.random.default_rng(n + deg + ef)
    x = rng.integers(0, 16, (n, 20)).astype(np.float32)
    l0 = np.zeros((n, deg + 1), np.uint32)
    l0[:, 0] = deg
    l0[:, 1:] = rng.integers(0, n, (n, deg))
    cols = rng.uniform(0, 1, (1, n))
    gi = GpuIndex(x, cols, l0=l0, device=0)
    q = rng.uniform(0, 16, (6, 20)).astype(np.float32).round(3)
    ent = rng.integers(0, n, 6)
    ids, dists, cnt, exh = gi.graph_batch(q, ent, [Cmp(0, "<", share)] * 6, ef,
                                          max_visited=max_visited)
    gi.close()
    lists = [l0[i, 1:].tolist() for i in range(n)]
    mask = cols[0] < share
    width = max(1, min(WMAX, 512 // deg))
    for i in range(6):
        want, w_exh = search(x.astype(np.float64), lists, q[i].astype(np.float64), int(ent[i]),
                             mask, ef, max_visited, width)
        assert cnt[i] == len(want) and bool(exh[i]) == w_exh
        np.testing.assert_allclose(dists[i, :len(want)], [w[0] for w in want], rtol=1e-5)
        if want:
            assert np.isin(ids[i, :len(want)], [w[1] for w in want]).mean() >= 0.99
