"""A CTA that gives up waits for its copies in flight first (bulk_drain,
fk_bulk.cuh): by reading, every early return of the midpoint kernel does; on
the device, the windows of a ring of barriers, in its first rounds and later,
whole or with one that never completes."""
import ctypes
import os
import re

import numpy as np
import pytest

import test_gpu_bulk as bulk

HERE = os.path.dirname(os.path.abspath(__file__))
WINDOW = 3 * 4 * 72


def test_every_early_return_of_the_midpoint_kernel_waits_for_its_windows():
    src = open(os.path.join(HERE, "..", "adjoint-optimization_b200", "csrc", "fk_run.cu")).read()
    body = src[src.index("void mid_run("):src.index("k_mid_run(")]
    body = body[body.index("fetch(k0);"):]
    returns = [m.start() for m in re.finditer(r"\breturn;", body)]
    assert len(returns) == 2
    for at in returns:
        assert "bulk_drain<3>(bar" in body[body.rindex("if (", 0, at):at]


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("drain") / "drain.so")
    old, bulk.PROBE = bulk.PROBE, os.path.join(HERE, "drain_probe.cu")
    try:
        bulk._build(out)
    finally:
        bulk.PROBE = old
    lib = ctypes.CDLL(out)
    lib.probe_drain.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint, ctypes.c_ulonglong, ctypes.c_void_p,
                                ctypes.POINTER(ctypes.c_float)]
    return lib


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [0, 16])
@pytest.mark.parametrize("total", [2, 3, 4, 7, 11])
def test_drain_waits_for_the_windows_in_flight(probe, total, extra):
    src = np.random.default_rng(total).standard_normal(total * WINDOW)
    out, ms = np.full(2 * WINDOW, np.nan), ctypes.c_float(0)
    assert probe.probe_drain(src.ctypes.data, total, extra, 50_000_000, out.ctypes.data, ctypes.byref(ms)) == 0
    np.testing.assert_array_equal(out, src[-2 * WINDOW:])
    if extra:
        assert 40.0 <= ms.value < 5000.0, ms.value  # the missing bytes: one bounded wait
    else:
        assert ms.value < 40.0, ms.value
