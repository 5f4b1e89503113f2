"""Sweeps of many steps in one launch (fk_run.cu) against one launch per step
(FKADJ_SWEEPS=0): the same arithmetic per cell, so the same bits, on grids at
the edges of every tile shape (one tile, one row or column of tiles, cut last
tiles, tiles of the least height, the largest grids that fit the device),
with frames at every remainder, and where the sweep has to give way: cells
between two holes, a source on every cell, a NaN among the inputs."""
import numpy as np
import pytest

from fkadj import _lib, api, workloads as W
from fkadj.batch import Batch
from test_gpu_edges import _custom

pytestmark = pytest.mark.gpu

SIZES = [(5, 7), (16, 16), (17, 33), (48, 64), (64, 200), (128, 128), (131, 97), (300, 40), (40, 610), (203, 331),
         (256, 256), (437, 501), (512, 512), (640, 400), (29 * 18, 64 * 8), (600, 700), (1031, 521)]


def _both(monkeypatch, call):
    out = []
    for v in ("0", "1"):
        monkeypatch.setenv("FKADJ_SWEEPS", v)
        out.append(call())
    return out


def _same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(a[~np.isnan(a)], b[~np.isnan(b)])


def _forward(inst, nstep, ghost=None, y0=None):
    return api.fk_forward_Et(inst.Et, inst.dt, inst.nt, inst.y0 if y0 is None else y0, inst.active_index, inst.ncols,
                             inst.nrows, inst.ghost if ghost is None else ghost, nstep, params=inst.params)[:2]


@pytest.mark.parametrize("rows,cols", SIZES)
def test_forward_sweep_gives_the_bits_of_single_steps(monkeypatch, rows, cols):
    inst = W.make_instance(rows, 23, ncols=cols, seed=rows + cols, n_obstacles=max(1, rows * cols // 2500),
                           intervals=5, r_range=(0.02, 0.1) if min(rows, cols) > 30 else (0.01, 0.02))
    (ys0, yf0), (ys1, yf1) = _both(monkeypatch, lambda: _forward(inst, 7))
    _same(ys0, ys1)
    _same(yf0, yf1)


@pytest.mark.parametrize("mode", [_lib.GRAD_REF, _lib.GRAD_EXACT])
@pytest.mark.parametrize("rows,cols", SIZES)
def test_gradient_sweeps_give_the_bits_of_single_steps(monkeypatch, rows, cols, mode):
    """37 steps: chunks of 16 (8), a short one, and sqrt segments of 7."""
    inst = W.make_instance(rows, 37, ncols=cols, seed=rows + cols, n_obstacles=max(1, rows * cols // 2500),
                           intervals=5, r_range=(0.02, 0.1) if min(rows, cols) > 30 else (0.01, 0.02), alpha=0.1)
    store = _lib.CKPT_SQRT if (rows + cols) % 2 else _lib.CKPT_FULL

    def call():
        with api.Problem(inst, opts=api.options(grad_mode=mode, ckpt_policy=store)) as pb:
            return pb.grad(inst.Et, inst.y0), pb.grad(inst.Et * 0.5)
    a, b = _both(monkeypatch, call)
    for x, y in zip(a, b):
        assert x["Lcost"] == y["Lcost"]
        assert np.abs(x["gradE"]).max() > 0
        assert np.array_equal(x["gradE"], y["gradE"])


@pytest.mark.parametrize("mode", [_lib.GRAD_REF, _lib.GRAD_EXACT])
@pytest.mark.parametrize("nt,budget", [(3, 4), (40, 4), (41, 9), (600, 60), (600, 200)])
def test_stores_and_windows(monkeypatch, mode, nt, budget):
    """Binomial and AUTO stores within `budget` states, horizons longer than the
    window of partial sums, and stage states kept or replayed (exact mode)."""
    inst = W.make_instance(40, nt, ncols=72, seed=nt, n_obstacles=4, intervals=3, objective="gradient")
    sb = 3 * 8 * 72 * 136
    out = {}
    for name, pol, b in (("full", _lib.CKPT_FULL, 0), ("auto", _lib.CKPT_AUTO, budget * sb),
                         ("binomial", _lib.CKPT_BINOMIAL, budget * sb), ("tight", _lib.CKPT_FULL, 2 * nt * sb)):
        def call():
            with api.Problem(inst, opts=api.options(grad_mode=mode, ckpt_policy=pol, ckpt_budget_bytes=b)) as pb:
                return pb.grad(inst.Et, inst.y0)["gradE"]
        a, c = _both(monkeypatch, call)
        assert np.array_equal(a, c), name
        out[name] = c
    for name in out:
        assert np.array_equal(out[name], out["full"]), name


def test_gradient_with_a_nan_input_is_a_numeric_error_either_way(monkeypatch):
    inst = W.make_instance(80, 20, ncols=100, seed=4, n_obstacles=3, intervals=4)
    y0 = inst.y0.copy()
    y0[inst.n_num // 2] = np.nan

    def call():
        with api.Problem(inst) as pb:
            with pytest.raises(_lib.FkadjError) as e:
                pb.grad(inst.Et, y0)
            good = pb.grad(inst.Et, inst.y0)["gradE"]  # the problem sweeps again
            return str(e.value), good
    a, b = _both(monkeypatch, call)
    assert a[0] == b[0]
    assert np.array_equal(a[1], b[1])


@pytest.mark.parametrize("nt", [3, 4, 5])
def test_shortest_sweeps_and_resident_state(monkeypatch, nt):
    inst = W.make_instance(96, nt, ncols=130, seed=nt, n_obstacles=6, intervals=3)

    def call():
        with api.Problem(inst) as pb:
            return [pb.objective(inst.Et, y, return_yf=True) for y in (inst.y0, None)]
    a, b = _both(monkeypatch, call)
    for x, y in zip(a, b):
        _same(x["yf"], y["yf"])
        assert x["Lcost"] == y["Lcost"]


def test_cells_between_two_holes(monkeypatch):
    mask = np.ones((70, 90), bool)
    mask[10, 10] = mask[12, 10] = False      # (11, 10): north and south are holes
    mask[20, 30] = mask[20, 32] = False      # (20, 31): west and east are holes
    mask[40, 41] = mask[40, 44] = mask[39, 43] = mask[41, 43] = False  # (40, 43) falls, then (40, 42)
    inst = _custom(mask, 30)
    (_, yf0), (_, yf1) = _both(monkeypatch, lambda: _forward(inst, 0))
    _same(yf0, yf1)
    u = yf1[:70 * 90].reshape(70, 90)
    assert np.isnan(u[40, 42]) and np.isnan(u[40, 43]) and np.isfinite(u[38, 42])


def test_source_on_every_cell(monkeypatch):
    inst = W.make_instance(120, 20, ncols=140, seed=3, n_obstacles=5, intervals=4)
    ghost = np.linspace(-1.0, 1.0, inst.ghost.size)
    (_, yf0), (_, yf1) = _both(monkeypatch, lambda: _forward(inst, 0, ghost=ghost))
    _same(yf0, yf1)


@pytest.mark.parametrize("field", [0, 1, 2])
def test_nan_input_stays_where_single_steps_keep_it(monkeypatch, field):
    """A NaN in an active cell: the per-step stencil takes it for a hole."""
    inst = W.make_instance(80, 20, ncols=100, seed=4, n_obstacles=3, intervals=4)
    y0 = inst.y0.copy()
    y0[field * inst.n_num + inst.n_num // 2] = np.nan
    (_, yf0), (_, yf1) = _both(monkeypatch, lambda: _forward(inst, 0, y0=y0))
    _same(yf0, yf1)


@pytest.mark.parametrize("mode", [_lib.GRAD_REF, _lib.GRAD_EXACT])
def test_pairs_of_the_binomial_store_on_a_grid_of_several_waves(mode):
    inst = W.make_instance(600, 9, ncols=700, seed=9, n_obstacles=100, intervals=3)
    sb = 3 * 8 * (640 + 8) * (704 + 8)

    def call(pol, b):
        with api.Problem(inst, opts=api.options(grad_mode=mode, ckpt_policy=pol, ckpt_budget_bytes=b)) as pb:
            return pb.grad(inst.Et, inst.y0)["gradE"]
    full = call(_lib.CKPT_FULL, 0)
    for states in (3, 4, 6):
        assert np.array_equal(call(_lib.CKPT_BINOMIAL, states * sb), full), states


@pytest.mark.parametrize("store", [_lib.CKPT_FULL, _lib.CKPT_SQRT])
@pytest.mark.parametrize("mode", [_lib.GRAD_REF, _lib.GRAD_EXACT])
def test_batched_sweeps_give_the_bits_of_single_problems(mode, store):
    """More problems than one launch takes, of two models, from one tile to the
    whole device and beyond; among them one without a gradient, one with cells
    between two holes (these fall, and the objective with them) and one with a
    NaN among its inputs."""
    sizes = [(5, 7), (16, 16), (300, 40), (40, 610), (131, 97), (512, 512), (600, 700), (256, 256), (64, 200)] + \
        [(48 + k, 64 + 3 * k) for k in range(12)]
    insts = [W.make_instance(r, 7 + 5 * (k % 9), ncols=c, dt=0.02 if k % 3 else 0.01, seed=k, intervals=4,
                             n_obstacles=max(1, r * c // 2500), alpha=0.1,
                             r_range=(0.02, 0.1) if min(r, c) > 30 else (0.01, 0.02))
             for k, (r, c) in enumerate(sizes)]
    mask = np.ones((70, 90), bool)
    mask[10, 10] = mask[12, 10] = False
    insts.append(_custom(mask, 30))
    bad = np.array(insts[4].y0)
    bad[insts[4].n_num // 2] = np.nan
    opts = api.options(grad_mode=mode, ckpt_policy=store)

    def single(x):
        with api.Problem(x, opts=opts) as pb:
            return pb.grad(x.Et, x.y0)
    want = [single(x) for x in insts[:-1]]
    with pytest.raises(_lib.FkadjError) as fallen:
        single(insts[-1])
    with Batch() as b:
        ids = [b.add_problem(x, grad_mode=mode, ckpt_policy=store) for x in insts]
        for repeat in range(2):
            jobs = [b.submit(p, x.Et, bad if k == 4 and repeat == 0 else x.y0, want_grad=k != 2)
                    for k, (p, x) in enumerate(zip(ids, insts))]
            b.run()
            with pytest.raises(_lib.FkadjError) as e:
                b.result(jobs[-1])
            assert e.value.status == fallen.value.status
            for k, (j, w) in enumerate(zip(jobs, want)):
                if k == 4 and repeat == 0:
                    with pytest.raises(_lib.FkadjError):
                        b.result(j)
                    continue
                r = b.result(j)
                assert r["Lcost"] == w["Lcost"], (k, repeat)
                if k != 2:
                    assert np.array_equal(r["gradE"], w["gradE"]), (k, repeat)
