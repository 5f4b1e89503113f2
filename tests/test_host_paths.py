"""Host paths that only a failing call reaches, run without a GPU: the
library's objects linked with a stand-in for the CUDA runtime
(fake_cudart.cpp) whose kernels do nothing, whose device memory can run out at
any allocation and whose cooperative launches can be refused.  Every buffer a
sweep is handed must lie in live device memory."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from fkadj import _lib, api, batch, serve, workloads as W
from fkadj.batch import Batch
from fkadj.serve import Server
from test_gpu_edges import _custom as custom_mask

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = _lib.PKG_DIR
MODES = [_lib.GRAD_REF, _lib.GRAD_EXACT]
STORES = [_lib.CKPT_FULL, _lib.CKPT_SQRT, _lib.CKPT_BINOMIAL]
FAULT_NAN = 2
ADMIT = "_ZN5fkadj12admit_sweepsElllll"
ESTIMATE = "_ZN5fkadj7Problem14estimate_bytesEiiiiliibb"


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    subprocess.run(["make", "-s", "-C", PKG, "-j4", "lib"], check=True)
    tmp = tmp_path_factory.mktemp("fake")
    obj, lib = str(tmp / "fake.o"), str(tmp / "libfkadj_fake.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", f"-I{cuda}/include", "-c", "-o", obj,
                    os.path.join(HERE, "fake_cudart.cpp")], check=True)
    objs = [os.path.join(PKG, "_build", f"fk_{n}.o")
            for n in ("kernels", "run", "engine", "spline", "noalloc", "batch", "serve", "matio")]
    # its own definitions of the runtime, whatever the process has loaded
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", lib, *objs, obj, "-lpthread", "-lz"],
                   check=True)
    return lib


@pytest.fixture
def fake(fake_path, monkeypatch):
    for v in ("FKADJ_SWEEPS", "FKADJ_TILES", "FKADJ_ADJ_PATH", "FKADJ_JCACHE", "FKADJ_ZGH_SEGMENTS",
              "FKADJ_SERVE_MODE", "FKADJ_SERVE_STREAMS", "FKADJ_ONESHOT_POOL"):
        monkeypatch.delenv(v, raising=False)
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", fake_path)
    monkeypatch.setattr(batch, "_bound", False)
    monkeypatch.setattr(serve, "_bound", False)
    L = _lib.load()
    for n in ("allocations", "in_use", "peak", "bad_spans"):
        getattr(L, f"fake_{n}").restype = C.c_int64
    L.fake_launches.restype = C.c_int64
    L.fake_launches.argtypes = [C.c_char_p]
    L.fake_first_bad.restype = C.c_char_p
    L.fake_reset.argtypes = [C.c_int64]
    L.fake_fail_allocations.argtypes = [C.c_int64, C.c_int64]
    L.fake_fail_host_allocation.argtypes = [C.c_int64]
    L.fake_fault.argtypes = [C.c_char_p, C.c_uint, C.c_int]
    _lib.check(L.fkadj_release_cached_memory())
    L.fake_reset(0)
    yield L
    assert L.fake_bad_spans() == 0, L.fake_first_bad().decode()
    L.fake_reset(0)


def _inst(rows=40, cols=72, nt=24, **kw):
    return W.make_instance(rows, nt, ncols=cols, seed=1, n_obstacles=3, intervals=3, alpha=0.1, **kw)


def _state_bytes(inst):
    return 3 * 8 * (-(-inst.nrows // 64) * 64 + 8) * (-(-inst.ncols // 64) * 64 + 8)


def _opts(inst, mode=_lib.GRAD_REF, store=_lib.CKPT_AUTO, states=0):
    return api.options(grad_mode=mode, ckpt_policy=store, ckpt_budget_bytes=int(states * _state_bytes(inst)))


def _sweeps(L):
    return L.fake_launches(b"k_fwd_run") + L.fake_launches(b"k_fwd_jobs")


@pytest.mark.parametrize("store", STORES)
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("rows,cols,nt", [(5, 7, 3), (40, 72, 24), (131, 97, 37), (300, 200, 70), (640, 900, 9)])
def test_sweeps_stay_in_their_buffers(fake, rows, cols, nt, mode, store):
    inst = _inst(rows, cols, nt)
    with api.Problem(inst, opts=_opts(inst, mode, store, 6 if store == _lib.CKPT_BINOMIAL else 0)) as pb:
        for y in (inst.y0, None):
            pb.grad(inst.Et, y, return_yf=True)
        pb.objective(inst.Et)
    if store != _lib.CKPT_BINOMIAL:
        with Batch() as b:
            ids = [b.add_problem(inst, grad_mode=mode, ckpt_policy=store) for _ in range(3)]
            for j in [b.submit(p, inst.Et, inst.y0, want_grad=k != 1) for k, p in enumerate(ids)]:
                b.run()
                b.result(j)
    assert fake.fake_launches(b"k_fwd_step") == 0 and fake.fake_launches(b"k_batch") == 0
    assert _sweeps(fake) > 0 or fake.fake_launches(b"k_fwd_tile") > 0


@pytest.mark.parametrize("sweeps,n_failing", [("1", 1), ("1", 1000), ("0", 1)])
@pytest.mark.parametrize("store", STORES[:2])
@pytest.mark.parametrize("mode", MODES)
def test_a_failed_allocation_leaves_no_missing_buffer(fake, monkeypatch, mode, store, sweeps, n_failing):
    """Allocations of a first gradient fail from any one on: the call gives its
    result without sweeps or reports the lack of memory, and the next one finds
    every buffer that a problem of its kind holds."""
    inst = _inst()
    opts = _opts(inst, mode, store)

    def held(v):
        monkeypatch.setenv("FKADJ_SWEEPS", v)
        before = fake.fake_in_use()
        with api.Problem(inst, opts=opts) as pb:
            fake.fake_fail_allocations(-1, 0)
            pb.grad(inst.Et, inst.y0)
            return fake.fake_in_use() - before, fake.fake_allocations()
    preset, swept = held("0"), held("1")
    monkeypatch.setenv("FKADJ_SWEEPS", sweeps)
    for k in range((swept if sweeps == "1" else preset)[1]):
        before = fake.fake_in_use()
        with api.Problem(inst, opts=opts) as pb:
            fake.fake_fail_allocations(k, n_failing)
            try:
                pb.grad(inst.Et, inst.y0)
            except _lib.FkadjError as e:
                assert e.status == _lib.ERR_NOMEM
            fake.fake_fail_allocations(-1, 0)
            pb.grad(inst.Et, inst.y0)
            runs = fake.fake_launches(b"k_adj_run")
            pb.grad(inst.Et)
            want = swept if fake.fake_launches(b"k_adj_run") > runs else preset
            assert fake.fake_in_use() - before >= want[0], k


@pytest.mark.parametrize("k", range(4))
def test_a_failed_change_of_the_store_is_made_again(fake, k):
    """The repeat after a NaN takes another store (no kept stage states); where
    its allocation fails, the next call must not take the old plan for done."""
    inst = _inst()
    with api.Problem(inst, opts=_opts(inst, _lib.GRAD_EXACT, _lib.CKPT_SQRT)) as pb:
        pb.grad(inst.Et, inst.y0)
        fake.fake_fault(b"k_fwd_run", FAULT_NAN, 1)
        fake.fake_fail_allocations(k, 1)
        try:
            pb.grad(inst.Et)
        except _lib.FkadjError as e:
            assert e.status == _lib.ERR_NOMEM
        fake.fake_fail_allocations(-1, 0)
        pb.grad(inst.Et)


@pytest.mark.parametrize("k", range(4))
def test_a_failed_pinned_allocation_leaves_no_missing_buffer(fake, k):
    inst = _inst()
    with api.Problem(inst) as pb:
        fake.fake_fail_host_allocation(k)
        try:
            pb.grad(inst.Et, inst.y0, return_yf=True)
        except _lib.FkadjError as e:
            assert e.status == _lib.ERR_NOMEM
        fake.fake_fail_host_allocation(-1)
        pb.grad(inst.Et, inst.y0, return_yf=True)
    with Server(hbm_budget_bytes=1 << 30) as sv:
        fake.fake_fail_host_allocation(k)
        rid = sv.submit(inst)
        try:
            sv.wait(rid)
        except _lib.FkadjError as e:
            assert e.status == _lib.ERR_NOMEM
        fake.fake_fail_host_allocation(-1)
        rid = sv.submit(inst)
        assert sv.wait(rid)


def _refused(fake, inst, call):
    runs = _sweeps(fake)
    with pytest.raises(_lib.FkadjError) as e:
        call()
    assert e.value.status == _lib.ERR_NOMEM
    assert _sweeps(fake) == runs and fake.fake_launches(b"k_fwd_step") == 0


@pytest.mark.parametrize("mode", MODES)
def test_a_refused_budget_leaves_the_sweeps_on(fake, mode):
    """A gradient whose store does not fit the caller's budget fails before
    any device work; the problem's objectives go on as sweeps."""
    inst = _inst()
    with api.Problem(inst, opts=_opts(inst, mode, _lib.CKPT_SQRT, 2)) as pb:
        for n in range(1, 3):
            _refused(fake, inst, lambda: pb.grad(inst.Et, inst.y0))
            pb.objective(inst.Et, inst.y0)
            assert _sweeps(fake) == n
    with Batch() as b:
        for states, store in ((2, _lib.CKPT_SQRT), (6, _lib.CKPT_BINOMIAL)):  # the latter is not a batch's
            p = b.add_problem(inst, grad_mode=mode, ckpt_policy=store, ckpt_budget_bytes=states * _state_bytes(inst))
            _refused(fake, inst, lambda: b.submit(p, inst.Et, inst.y0))
            runs = _sweeps(fake)
            j = b.submit(p, inst.Et, inst.y0, want_grad=False)
            b.run()
            b.result(j)
            assert _sweeps(fake) > runs and fake.fake_launches(b"k_batch_fwd") == 0


@pytest.mark.parametrize("mode", MODES)
def test_sweeps_come_back_where_the_preset_kernels_lacked_memory_too(fake, mode):
    inst = _inst()
    with api.Problem(inst, opts=_opts(inst, mode, _lib.CKPT_SQRT)) as pb:
        fake.fake_fail_allocations(0, 1000)
        with pytest.raises(_lib.FkadjError) as e:
            pb.grad(inst.Et, inst.y0)
        assert e.value.status == _lib.ERR_NOMEM
        fake.fake_fail_allocations(-1, 0)
        steps = fake.fake_launches(b"k_fwd_step")
        pb.grad(inst.Et, inst.y0)
        assert fake.fake_launches(b"k_adj_run") > 0 and fake.fake_launches(b"k_fwd_step") == steps


@pytest.mark.parametrize("want_grad", [True, False])
@pytest.mark.parametrize("store", STORES[:2])
@pytest.mark.parametrize("mode", MODES)
def test_a_batched_job_that_cannot_be_repeated_fails_alone(fake, mode, store, want_grad):
    """A NaN among one job's inputs, and no memory for the tick kernels'
    buffers: that job reports it, the others give their results, and both
    problems take new jobs (as sweeps)."""
    inst = _inst()
    with Batch() as b:
        ids = [b.add_problem(inst, grad_mode=mode, ckpt_policy=store) for _ in range(2)]
        jobs = [b.submit(ids[0], inst.Et, inst.y0, want_grad=want_grad), b.submit(ids[1], inst.Et, inst.y0)]
        fake.fake_fault(b"k_fwd_jobs", FAULT_NAN, 1)  # the first problem's
        while not b.done(jobs[1]):
            b.tick()
            fake.fake_fail_allocations(0, 1000)
        if want_grad:
            with pytest.raises(_lib.FkadjError) as e:
                b.run()
                b.result(jobs[0])
            assert e.value.status == _lib.ERR_NOMEM
        else:  # an objective needs no more buffers
            b.run()
            b.result(jobs[0])
        b.result(jobs[1])
        fake.fake_fail_allocations(-1, 0)
        ticks = fake.fake_launches(b"k_batch")
        for j in [b.submit(p, inst.Et, inst.y0) for p in ids]:
            b.run()
            assert b.result(j)["gradE"].size == inst.nt + 1
        assert fake.fake_launches(b"k_batch") == ticks


@pytest.mark.parametrize("store", STORES)
@pytest.mark.parametrize("mode", MODES)
def test_a_repeat_without_memory_takes_the_sweeps_buffers(fake, mode, store):
    inst = _inst()
    with api.Problem(inst, opts=_opts(inst, mode, store, 6 if store == _lib.CKPT_BINOMIAL else 0)) as pb:
        pb.grad(inst.Et, inst.y0)
        for _ in range(2):
            runs = fake.fake_launches(b"k_adj_run")
            fake.fake_fault(b"k_fwd_run", FAULT_NAN, 1)
            fake.fake_fail_allocations(0, 1)
            pb.grad(inst.Et)
            fake.fake_fail_allocations(-1, 0)
            pb.grad(inst.Et)
            assert fake.fake_launches(b"k_adj_run") >= runs + 2


@pytest.mark.parametrize("store", STORES[:2])
@pytest.mark.parametrize("mode", MODES)
def test_a_refused_cooperative_launch_gives_way_to_tile_kernels(fake, mode, store):
    """A stream that sees fewer SMs than the device has refuses a CTA per SM."""
    inst = _inst()
    fake.fake_refuse_cooperative(1)
    call = (inst.Et, inst.dt, inst.nt, inst.y0, inst.active_index, inst.ncols, inst.nrows, inst.ghost)
    api.fk_forward_Et(*call, 5, params=inst.params)
    api.fk_grad_Et(*call, inst.gamma, inst.S, inst.alpha, params=inst.params, opts=_opts(inst, mode, store))
    with api.Problem(inst, opts=_opts(inst, mode, store)) as pb:
        pb.grad(inst.Et, inst.y0)
        steps = fake.fake_launches(b"k_fwd_tile")
        pb.objective(inst.Et)
        assert fake.fake_launches(b"k_fwd_tile") == steps + inst.nt
    with Batch() as b:
        jobs = [b.submit(b.add_problem(inst, grad_mode=mode, ckpt_policy=store), inst.Et, inst.y0, want_grad=k > 0)
                for k in range(3)]
        b.run()
        jobs.append(b.submit(b.add_problem(inst, grad_mode=mode, ckpt_policy=store), inst.Et, inst.y0))
        b.run()
        for j in jobs:
            b.result(j)
    assert fake.fake_launches(b"k_adj_tile") > 0
    assert _sweeps(fake) == 0 and fake.fake_launches(b"k_fwd_step") == 0 and fake.fake_launches(b"k_batch") == 0


def test_a_server_stops_while_its_workers_go_to_sleep(fake_path, tmp_path):
    """In a process of its own, which must end."""
    slow = str(tmp_path / "slow_wait.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-o", slow, os.path.join(HERE, "slow_wait.cpp"), "-ldl"], check=True)
    code = ("import time\n"
            "from fkadj.serve import Server\n"
            "sv = Server(hbm_budget_bytes=1 << 30)\n"
            "time.sleep(0.02)\n"
            "sv.close()\n")
    env = dict(os.environ, FKADJ_LIB=fake_path, LD_PRELOAD=slow, PYTHONPATH=PKG, OPENBLAS_NUM_THREADS="1")
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=60)


@pytest.mark.parametrize("mask", ["open", "pinched"])
@pytest.mark.parametrize("nan", [False, True])
@pytest.mark.parametrize("store", STORES[:2])
@pytest.mark.parametrize("mode", MODES)
def test_a_served_request_stays_within_the_budget(fake, monkeypatch, mode, store, nan, mask):
    """The server's estimate bounds the device memory a request takes, with
    sweeps or without (a cell between two holes), repeated after a NaN or not,
    for budgets from the least that holds the estimate on; on a large grid with
    a short horizon the partial sums' window is what counts."""
    estimate = getattr(fake, ESTIMATE)
    estimate.restype = C.c_int64
    estimate.argtypes = [C.c_int] * 4 + [C.c_int64, C.c_int, C.c_int, C.c_bool, C.c_bool]
    for rows, cols, nt in ((40, 72, 24), (131, 97, 90), (640, 500, 24)):
        if mask == "pinched":
            m = np.ones((rows, cols), bool)
            m[10, 10] = m[12, 10] = False
            inst = custom_mask(m, nt)
        else:
            inst = _inst(rows, cols, nt)
        least = [estimate(rows, cols, nt, inst.n_num, inst.S.nnz, mode, store, g, False) for g in (True, False)]
        for budget in [least[0], least[0] + 5 * _state_bytes(inst), 2 * least[0], 8 * least[0]]:
            with Server(opts=_opts(inst, mode, store), hbm_budget_bytes=budget) as sv:
                for grad in (True, False):
                    _lib.check(fake.fkadj_release_cached_memory())
                    fake.fake_reset(0)
                    base = fake.fake_in_use()
                    if nan:
                        fake.fake_fault(b"k_fwd_", FAULT_NAN, 1)
                    assert sv.wait(sv.submit(inst, want_grad=grad), 60)
                    assert fake.fake_peak() - base <= budget, (rows, cols, nt, budget / least[0], grad)
                assert sv.stats["failed"] == 0


@pytest.mark.parametrize("budget,used,est,est_sweeps,following,want", [
    (100, 0, 40, 60, -1, True), (100, 0, 40, 100, -1, True), (100, 0, 40, 101, -1, False),
    (100, 40, 40, 60, -1, True), (100, 41, 40, 60, -1, False),
    (100, 0, 40, 60, 40, True),     # both fit
    (100, 0, 40, 61, 40, False),    # the next one fits beside the preset kernels only
    (100, 0, 40, 61, 61, True)])    # the next one waits either way
def test_sweeps_do_not_keep_the_next_request_out(fake, budget, used, est, est_sweeps, following, want):
    admit = getattr(fake, ADMIT)
    admit.restype = C.c_bool
    admit.argtypes = [C.c_int64] * 5
    assert admit(budget, used, est, est_sweeps, following) == want


@pytest.mark.parametrize("rows,cols,nt,mode,states,want", [
    (256, 256, 400, 0, 40, "sqrt"), (256, 256, 400, 0, 395, "sqrt"), (256, 256, 400, 1, 40, "sqrt"),
    (256, 256, 400, 1, 200, "sqrt"), (512, 512, 400, 0, 40, "sqrt"), (512, 512, 400, 1, 40, "sqrt"),
    (512, 512, 400, 1, 100, "sqrt"), (700, 600, 300, 0, 35, "sqrt"), (700, 600, 300, 1, 35, "binomial"),
    (1024, 768, 200, 0, 29, "sqrt"), (1024, 768, 200, 1, 66, "binomial"), (256, 256, 400, 0, 39, "binomial"),
    (128, 128, 600, 1, 300, "sqrt"), (400, 380, 300, 1, 100, "sqrt"), (48, 64, 130, 1, 30, "binomial"),
    (40, 72, 24, 0, 24, "sqrt"), (40, 72, 24, 0, 25, "full")])
def test_auto_takes_the_store_that_sweeps_cost_less(fake, rows, cols, nt, mode, states, want):
    """The faster of the two by more than 3 % where both were measured
    (binomial_step_cost), but for differences below 2 ms on small grids; a store
    that does not fit is not taken."""
    inst = _inst(rows, cols, nt)
    with api.Problem(inst, opts=_opts(inst, mode, _lib.CKPT_AUTO, states)) as pb:
        pb.grad(inst.Et, inst.y0)
        assert pb.last_plan["policy"] == want


def test_a_problem_without_memory_for_the_flags_or_the_exchange_is_made_all_the_same(fake, monkeypatch):
    """What the preset kernels need is asked for; nothing is left behind where that fails."""
    inst = _inst()

    def made(k):
        before = fake.fake_in_use()
        fake.fake_fail_allocations(k, 1)
        try:
            with api.Problem(inst) as pb:
                n = fake.fake_allocations()
                fake.fake_fail_allocations(-1, 0)
                pb.grad(inst.Et, inst.y0)
                return n
        except _lib.FkadjError as e:
            assert e.status == _lib.ERR_NOMEM
        finally:
            fake.fake_fail_allocations(-1, 0)
            assert fake.fake_in_use() == before
    monkeypatch.setenv("FKADJ_SWEEPS", "0")
    preset = made(-1)
    monkeypatch.delenv("FKADJ_SWEEPS")
    swept = made(-1)
    assert swept == preset + 2
    assert sum(made(k) is not None for k in range(swept)) == 2


@pytest.mark.parametrize("mode", MODES)
def test_the_lattice_of_a_swept_problem_stays_what_it_was_made_with(fake, monkeypatch, mode):
    """FKADJ_ZGH_SEGMENTS=0 keeps a problem made under it from sweeping; set
    later, it must not shrink the rows that the sweeps write."""
    inst = _inst()
    with api.Problem(inst, opts=_opts(inst, mode)) as pb:
        monkeypatch.setenv("FKADJ_ZGH_SEGMENTS", "0")
        pb.grad(inst.Et, inst.y0)
        assert fake.fake_launches(b"k_adj_run") > 0
