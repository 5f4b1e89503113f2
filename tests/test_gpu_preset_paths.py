"""The launches that problems without sweeps run (FKADJ_SWEEPS=0 here; grids
with a cell between two holes, fixed presets, the repeat after a NaN and short
memory elsewhere): gradients replayed as graphs, segment graphs, ticks as
graphs, served requests.  The comparisons are those of the modules named, which
by default compare sweeps with sweeps; each call must have launched a kernel
per step.  And the other way round: where sweeps are to run they do, once."""
import numpy as np
import pytest

from fkadj import _lib, api, workloads as W
from fkadj.batch import Batch
import test_gpu_batch as batches
import test_gpu_graphs as graphs
import test_gpu_serve as served

pytestmark = pytest.mark.gpu
MODES = [_lib.GRAD_REF, _lib.GRAD_EXACT]


@pytest.fixture
def calls(monkeypatch):
    """(launches, steps) of every gradient and batch from here on."""
    monkeypatch.setenv("FKADJ_SWEEPS", "0")
    seen = []
    grad, run = api.Problem.grad, Batch.run

    def grad_(self, *a, **k):
        r = grad(self, *a, **k)
        seen.append((self.last_launches, self.nt))
        return r

    def run_(self):
        before = self.stats["launches"]
        run(self)
        seen.append((self.stats["launches"] - before, max(self._nt.values())))
    monkeypatch.setattr(api.Problem, "grad", grad_)
    monkeypatch.setattr(Batch, "run", run_)
    yield seen
    assert all(n >= steps for n, steps in seen), seen


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("ckpt,budget", [(_lib.CKPT_FULL, 0), (_lib.CKPT_SQRT, 0), (_lib.CKPT_BINOMIAL, 6)])
def test_graph_replay(calls, mode, ckpt, budget):
    graphs.test_graph_replay_is_bit_identical_to_plain_launches(mode, ckpt, budget)
    assert len(calls) == 6


def test_profiled_launches(calls):
    graphs.test_profiling_and_graph_runs_agree()
    assert len(calls) == 3


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("nt", [120, 97])
def test_segment_graphs(calls, monkeypatch, mode, nt):
    """Of the drop-in call and, with its launches counted, of a problem's first gradient."""
    graphs.test_one_shot_segment_graphs_are_bit_identical(monkeypatch, mode, nt)
    inst = W.make_instance(64, nt, seed=82, n_obstacles=5, intervals=12, ncols=80, objective="gradient", alpha=0.1)
    out = []
    for v in ("0", "1"):
        monkeypatch.setenv("FKADJ_SEGMENT_GRAPHS", v)
        with api.Problem(inst, opts=api.options(grad_mode=mode, ckpt_policy=_lib.CKPT_SQRT)) as pb:
            out.append(pb.grad(inst.Et, inst.y0)["gradE"])
    assert np.array_equal(out[0], out[1]) and len(calls) == 2


@pytest.mark.parametrize("mode", MODES)
def test_tick_graphs(calls, monkeypatch, mode):
    batches.test_tick_blocks_replayed_as_graphs_give_the_bits_of_single_ticks(monkeypatch, mode)
    assert len(calls) == 2


def test_presets_set_between_ticks(calls, monkeypatch):
    batches.test_presets_set_after_objective_only_ticks(monkeypatch)
    assert len(calls) == 1


@pytest.mark.parametrize("mode", ["streams", "ticks"])
def test_served_requests(calls, monkeypatch, mode):
    served.test_served_results_match_one_shot_and_are_mix_invariant(monkeypatch, mode)


@pytest.mark.parametrize("store", [_lib.CKPT_FULL, _lib.CKPT_SQRT])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("rows,cols,fits", [(5, 7, True), (64, 200, True), (131, 97, True), (437, 501, True),
                                            (512, 512, True), (600, 700, False), (1031, 521, False)])
def test_sweeps_run_and_are_not_repeated(monkeypatch, rows, cols, fits, mode, store):
    """One launch for many steps where the grid's tiles fit the device, one
    forward and one backward launch a step beyond; the preset kernels, also of
    a repeat after a NaN, launch three a step."""
    monkeypatch.delenv("FKADJ_SWEEPS", raising=False)
    inst = W.make_instance(rows, 60, ncols=cols, seed=rows + cols, n_obstacles=max(1, rows * cols // 2500),
                           intervals=5, r_range=(0.02, 0.1) if min(rows, cols) > 30 else (0.01, 0.02), alpha=0.1)
    with api.Problem(inst, opts=api.options(grad_mode=mode, ckpt_policy=store)) as pb:
        pb.objective(inst.Et, inst.y0)
        assert pb.last_launches < 12 if fits else inst.nt <= pb.last_launches < inst.nt + 12
        pb.grad(inst.Et)
        recomputed = pb.last_plan["recompute_steps"] + 60 // 8 if store == _lib.CKPT_SQRT else 0
        assert pb.last_launches < 60 if fits else pb.last_launches < 2 * inst.nt + recomputed + 50
