"""A wait that runs out in any scan of the graph builder fails the build: the
batches of an insertion step clear and move one another's watchdog word."""
import ctypes as C

import numpy as np
import pytest

from paves_b200 import _lib

pytestmark = pytest.mark.gpu


def build(x, wait_ns, batch):
    L = _lib.lib()
    err = C.create_string_buffer(256)
    n, d = x.shape
    h = L.pv_hnsw_build_gpu_wait(_lib.ptr(x), n, d, 8, 31, 0, _lib.FV_GPU_PREC_BF16, wait_ns,
                                 batch, err, 256)
    if h:
        L.pv_hnsw_free(h)
    return bool(h), err.value.decode()


# 20,000 rows: scans 0-6 are steps of one batch each, 7-8, 9-12 and 13-14
# (the last of 1568 rows) steps of several
@pytest.mark.parametrize("batch", [6, 7, 8, 9, 11, 12, 13, 14])
def test_an_expired_wait_fails_the_build(batch):
    x = np.random.default_rng(0).integers(0, 200, (20_000, 64)).astype(np.float32)
    ok, err = build(x, 1, batch)  # 1 ns: every wait that must wait expires
    assert not ok and "wait expired" in err
    assert build(x, 0, batch) == (True, "")


def test_limits():
    x = np.zeros((100, 16), np.float32)
    assert not build(x, 20_000_000_000, 0)[0]
    assert build(x, 1, 99)[0]  # no such scan
