"""Three short-list groups are for tables in no order, whoever asks: a saved
plan that names them for rows stored cluster by cluster runs with whole
lists, and the tuner leaves them out."""
import numpy as np
import pytest

from paves_b200 import GpuIndex, _lib
from paves_b200.stream import Stream

pytestmark = pytest.mark.gpu


def rows(n, dim, per, seed):
    rng = np.random.default_rng(seed)
    c = rng.integers(40, 200, (-(-n // per), dim))
    x = np.repeat(c, per, 0)[:n] + rng.integers(-9, 10, (n, dim))
    return x.astype(np.float32), rng


def test_ordered_rows(tmp_path):
    n, dim, k, nb = 80_000, 128, 16, 256  # supersets of 64: lists of 64 hold them, of 32 do not
    x, rng = rows(n, dim, 128, 5)
    q = x[rng.integers(0, n, nb)] + rng.integers(-2, 3, (nb, dim)).astype(np.float32)
    gi = GpuIndex(x, None, device=0, precision=_lib.FV_GPU_PREC_BF16)
    path = str(tmp_path / "tune.txt")
    s = Stream(gi, nb, k, q, path)
    plans = s.plans()
    s.close()
    assert all(p["epi"] < 3 for p in plans)
    with open(path) as f:  # the same file with three groups in every plan
        lines = [ln.split() for ln in f]
    for ln in lines:
        if ln[6] == str(_lib.PV_MODE_LOW):
            ln[7], ln[8] = "3", "3"
    with open(path, "w") as f:
        f.writelines(" ".join(ln) + "\n" for ln in lines)
    s = Stream(gi, nb, k, q, path)
    assert any(p["epi"] == 3 for p in s.plans())
    ids, dists, cnt, _ = s.run(q, [None] * nb, k)
    last = s.last()
    s.close()
    gi.close()
    assert last == {"uncertain": 0, "fallback": 0}
    ex = GpuIndex(x, None, device=0)
    assert _lib.lib().pv_exact_tc(ex.handle, 0) == 0
    i2, d2, c2, _ = ex.brute_batch(q, [None] * nb, k)
    ex.close()
    assert np.array_equal(cnt, c2) and np.array_equal(ids, i2) and np.array_equal(dists, d2)
