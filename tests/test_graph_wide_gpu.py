"""Graph search over rows of thousands of dims: as the same rows without
their zero dims."""
import numpy as np
import pytest

from paves_b200 import GpuError, GpuIndex
from paves_b200.pred import Cmp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [8000, 8440, 9000, 11460])
def test_same_as_the_narrow_rows(dim):
    rng = np.random.default_rng(1)
    n, nq, deg = 1500, 5, 16
    x = rng.integers(0, 32, (n, 64)).astype(np.float32)
    q = rng.integers(0, 32, (nq, 64)).astype(np.float32)
    l0 = np.zeros((n, deg + 1), np.uint32)
    l0[:, 0] = deg
    l0[:, 1:] = rng.integers(0, n, (n, deg))
    cols = rng.uniform(0, 1, (1, n))
    ent = rng.integers(0, n, nq)
    res = []
    for pad in (0, dim - 64):
        gi = GpuIndex(np.pad(x, ((0, 0), (0, pad))), cols, l0=l0, device=0)
        res.append(gi.graph_batch(np.pad(q, ((0, 0), (0, pad))), ent, [Cmp(0, "<", 0.3)] * nq, 32))
        gi.close()
    for a, b in zip(*res):
        assert np.array_equal(a, b)


def test_more_dims_are_refused():
    x, l0 = np.zeros((4, 11464), np.float32), np.tile(np.uint32([1, 0]), (4, 1))
    gi = GpuIndex(x, None, l0=l0, device=0)
    with pytest.raises(GpuError):
        gi.graph_batch(x[:1], [0], [None], 4)
    gi.close()
