"""Lists longer than a search step takes in are gone through in several."""
import numpy as np
import pytest

from paves_b200 import GpuIndex
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deg", [512, 513, 600, 1024, 1500])
def test_star(deg):
    n = deg + 1
    rng = np.random.default_rng(deg)
    x = rng.integers(0, 50, (n, 24)).astype(np.float32)
    l0 = np.zeros((n, deg + 1), np.uint32)
    l0[0, 0], l0[0, 1:] = deg, np.arange(1, n)  # the rest points back at row 0
    l0[1:, 0] = 1
    cols = np.arange(n, dtype=np.float64)[None]
    gi = GpuIndex(x, cols, l0=l0, device=0)
    ids, _, cnt, exh = gi.graph_batch(x[:2], [0, 0], [Cmp(0, ">=", float(n - 40))] * 2, 64)
    gi.close()
    assert (exh == 1).all() and (cnt == 40).all()
    assert np.array_equal(np.sort(ids[:, :40]), np.tile(np.arange(n - 40, n), (2, 1)))
