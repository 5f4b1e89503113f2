"""Drop-in calls from several threads at once: each takes its own stream,
events and pinned blocks from what earlier calls left, and gives them back;
every result has the bits of the call made alone, before and after the kept
memory is handed back."""
import threading

import numpy as np
import pytest

from fkadj import _lib, api, workloads as W

pytestmark = pytest.mark.gpu

INSTS = [W.make_instance(r, nt, ncols=c, seed=r + c, n_obstacles=4, intervals=6, alpha=0.1)
         for r, c, nt in ((40, 56, 60), (96, 64, 90), (128, 128, 40), (203, 131, 30), (64, 200, 50))]


def _calls(inst, mode):
    call = (inst.Et, inst.dt, inst.nt, inst.y0, inst.active_index, inst.ncols, inst.nrows, inst.ghost)
    ys, yf, _ = api.fk_forward_Et(*call, 7, params=inst.params)
    g = api.fk_grad_Et(*call, inst.gamma, inst.S, inst.alpha, params=inst.params,
                       opts=api.options(grad_mode=mode, ckpt_policy=_lib.CKPT_SQRT), return_yf=True)
    return np.nan_to_num(ys), np.nan_to_num(yf), g[0], np.array(g[1:4]), np.nan_to_num(g[5])


def test_calls_at_once_give_the_bits_of_calls_alone():
    want = [[_calls(i, m) for m in (_lib.GRAD_REF, _lib.GRAD_EXACT)] for i in INSTS]
    errors = []

    def client(t):
        try:
            for k in range(12):
                i, m = (t + k) % len(INSTS), (t + k // 2) % 2
                for a, b in zip(_calls(INSTS[i], m), want[i][m]):
                    assert np.array_equal(a, b), (t, k)
        except BaseException as e:  # noqa: B902
            errors.append(e)
    for _ in range(2):
        threads = [threading.Thread(target=client, args=(t,)) for t in range(12)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(300)
        assert not any(t.is_alive() for t in threads) and not errors, errors
        api.release_cached_memory()
