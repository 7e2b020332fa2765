"""Streams over rows stored cluster by cluster: the tuner counts what a plan
leaves uncertified (those queries are run again), and saved plans run as they
are; the answers are the exact scan's."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.stream import Stream

pytestmark = pytest.mark.gpu
BF16 = _lib.FV_GPU_PREC_BF16


def rows(n, dim, per, seed):
    rng = np.random.default_rng(seed)
    c = rng.integers(40, 200, (-(-n // per), dim))
    x = np.repeat(c, per, 0)[:n] + rng.integers(-9, 10, (n, dim))
    return x.astype(np.float32), rng


def exact(x, q, k):
    gi = GpuIndex(x, None, device=0)
    assert _lib.lib().pv_exact_tc(gi.handle, 0) == 0
    r = gi.brute_batch(q, [None] * len(q), k)
    gi.close()
    return r


def run(s, q, k, want):
    ids, dists, cnt, _ = s.run(q, [None] * len(q), k)
    assert s.last()["fallback"] == 0
    assert np.array_equal(cnt, want[2]) and np.array_equal(ids, want[0])
    assert np.array_equal(dists, want[1])
    return s.last()["uncertain"]


def test_saved_three_groups(tmp_path):
    n, dim, k, nb = 80_000, 128, 16, 256  # supersets of 64: lists of 64 hold them, of 32 do not
    x, rng = rows(n, dim, 128, 5)
    q = x[rng.integers(0, n, nb)] + rng.integers(-2, 3, (nb, dim)).astype(np.float32)
    want = exact(x, q, k)
    gi = GpuIndex(x, None, device=0, precision=BF16)
    path = str(tmp_path / "tune.txt")
    s = Stream(gi, nb, k, q, path)
    assert run(s, q, k, want) == 0
    s.close()
    with open(path) as f:  # the same file with three groups in every plan
        lines = [ln.split() for ln in f]
    for ln in lines:
        if ln[6] == str(_lib.PV_MODE_LOW):
            ln[7], ln[8] = "3", "3"
    with open(path, "w") as f:
        f.writelines(" ".join(ln) + "\n" for ln in lines)
    s = Stream(gi, nb, k, q, path)
    assert any(p["epi"] == 3 for p in s.plans())
    run(s, q, k, want)
    s.close()
    gi.close()


def test_plans_that_flag_are_charged(tmp_path):
    """A cluster of 9,000 rows that all lie within the sample's bound: three
    groups' runs are full and flag every query, whole lists none."""
    rng = np.random.default_rng(2)
    n, dim, nb, k = 150_000, 64, 512, 16
    x = rng.integers(0, 200, (n, dim)).astype(np.float32)
    x[30_000:39_000] = 100 + rng.integers(-3, 4, (9000, dim))
    q = (100 + rng.integers(-3, 4, (nb, dim))).astype(np.float32)
    want = exact(x, q, k)
    gi = GpuIndex(x, None, device=0, precision=BF16)
    s = Stream(gi, nb, k, q, str(tmp_path / "t.txt"))
    assert run(s, q, k, want) == 0
    s.close()
    gi.close()
