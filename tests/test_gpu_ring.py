"""The sweeps' edge exchange (fk_ring.cuh) on one CTA: the ring around a tile
takes its neighbours' values of the step asked for, cells outside the grid's
tiles stay as they are; a value that never comes ends the wait at its limit,
another CTA's fault at once, and the context stays usable."""
import ctypes

import numpy as np
import pytest

import test_gpu_bulk as bulk

HALO, TX, TY = 4, 16, 5
RW, LD, ROWS = TX + 8, 3 * TX + 8, 3 * TY + 8
TAG = 7


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ring") / "ring.so")
    old, bulk.PROBE = bulk.PROBE, bulk.PROBE.replace("bulk_probe", "ring_probe")
    try:
        bulk._build(out)
    finally:
        bulk.PROBE = old
    lib = ctypes.CDLL(out)
    lib.probe_ring.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_ulonglong, ctypes.c_void_p,
                               ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]

    def run(x, by, bx, fault=0):
        out = np.empty((3, TY + 8, RW))
        status, f, ms = np.zeros(1, np.int32), np.array([fault], np.uint32), np.zeros(1, np.float32)
        rc = lib.probe_ring(x.ctypes.data, by, bx, TAG, out.ctypes.data, status.ctypes.data, f.ctypes.data,
                            ms.ctypes.data)
        assert rc == 0, f"CUDA error {rc}"
        return out, status[0], f[0], ms[0]
    return run


def _exchange():
    x = np.zeros((3, ROWS, LD), dtype=[("v", np.float64), ("tag", np.uint64)])
    x["v"] = np.arange(x.size).reshape(x.shape)
    x["tag"] = TAG
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("by,bx", [(1, 1), (0, 0), (2, 2), (0, 1), (1, 2)])
def test_ring_takes_the_neighbours_values(probe, by, bx):
    x = _exchange()
    out, status, fault, _ = probe(x, by, bx)
    want = x["v"][:, by * TY:by * TY + TY + 8, bx * TX:bx * TX + RW].copy()
    i = np.arange(TY + 8)[:, None] + by * TY - HALO
    j = np.arange(RW)[None, :] + bx * TX - HALO
    inside = (i >= by * TY) & (i < by * TY + TY) & (j >= bx * TX) & (j < bx * TX + TX)
    want[:, inside | (i < 0) | (i >= 3 * TY) | (j < 0) | (j >= 3 * TX)] = -1.0
    assert status == 1 and fault == 0
    np.testing.assert_array_equal(out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("field,row,col", [(0, 0, 0), (2, 3, 23), (1, 4 + TY, 12), (2, 4 + TY + 3, 0)])
def test_a_value_that_never_comes_ends_the_wait(probe, field, row, col):
    x = _exchange()
    x["tag"][field, TY + row, TX + col] = TAG - 2  # the middle tile's window
    _, status, fault, ms = probe(x, 1, 1)
    assert status == 0 and fault == 1
    assert 40.0 <= ms < 5000.0, ms
    _, status, fault, ms = probe(x, 1, 1, fault=1)  # another CTA gave up
    assert status == 0 and fault == 1 and ms < 40.0, ms
    _, status, fault, _ = probe(_exchange(), 1, 1, fault=2)  # a NaN elsewhere does not end it
    assert status == 1 and fault == 2
