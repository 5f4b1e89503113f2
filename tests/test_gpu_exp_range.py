"""The kernels' exponential far outside the model's range: within its
documented one (|16 x / ln 2| < 2^31) it saturates in the argument's
direction."""
import ctypes

import numpy as np
import pytest

import test_gpu_mathfn as mathfn


@pytest.mark.gpu
def test_the_exponential_saturates_in_the_arguments_direction(tmp_path):
    lib = ctypes.CDLL(mathfn._build(str(tmp_path / "probe.so")))
    lib.probe_exp.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_longlong]
    end = 2.0 ** 31 * np.log(2.0) / 16.0
    x = np.array([693.0, 710.0, 1e4, 3.3e5, 1e7, 0.999 * end])
    x = np.concatenate([x, -x - 20.0])
    own, ref = np.empty_like(x), np.empty_like(x)
    assert lib.probe_exp(x.ctypes.data, own.ctypes.data, ref.ctypes.data, x.size) == 0
    up, down = own[:6], own[6:]
    # m clamped to its ends, 2^(j/16) in [1, 2), e^(f ln2/16) within 2^(+-1/32)
    assert np.all(up >= 2.0 ** (998 - 1 / 32)) and np.all(up < 2.0 ** (999 + 1 / 32)), up
    assert np.all(down >= 2.0 ** (-1020 - 1 / 32)) and np.all(down < 2.0 ** (-1019 + 1 / 32)), down
