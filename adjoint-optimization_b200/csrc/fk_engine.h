// fk_engine.h -- resident FK problem: geometry, objective, work buffers and
// the trajectory store of one instance on one GPU, plus the forward and
// gradient drivers (the roles of fk_forward_Et_comp, cu-F:646-849, and
// fk_grad_Et_comp, cu-G:1569-1938).
#pragma once

#include <cstdint>
#include <functional>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/fkadj.h"
#include "fk_kernels.h"
#include "fk_run.h"
#include "fk_spline.h"

namespace fkadj {

void set_error(const std::string& msg);

// One device allocation released on destruction.  With a memory pool set
// (problems owned by a batch engine) allocation and release are stream-ordered
// on `st`: releasing needs no device synchronisation, so a finished request can
// free its memory while the others keep running.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaStream_t st = nullptr;
    cudaMemPool_t pool = nullptr;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) {
            if (pool) cudaFreeAsync(p, st);
            else cudaFree(p);
        }
        p = nullptr;
        bytes = 0;
    }
    cudaError_t alloc(size_t b) {
        release();
        if (b == 0) return cudaSuccess;
        cudaError_t e = pool ? cudaMallocFromPoolAsync(&p, b, pool, st) : cudaMalloc(&p, b);
        if (e == cudaSuccess) bytes = b;
        else p = nullptr;
        return e;
    }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

struct Timing {
    double fwd_ms = 0, bwd_ms = 0, total_ms = 0;
};

// Where the states y(t_i) live during one gradient.
struct TrajPlan {
    int policy = FKADJ_CKPT_FULL;  // resolved policy (FULL / SQRT / BINOMIAL)
    int stride = 1;                // steps between stored states (SQRT)
    int nslots = 0;                // stored state slots
    int seg_slots = 0;             // recompute buffer slots
    bool keep_f = false;           // kept beside the states the backward sweep walks (FULL: all,
                                   // SQRT: the segment): k1 = f(y_t, Et[t]) (reference mode, per-step
                                   // launches) or the three stage states (exact mode, sweeps)
    int64_t recompute = 0;         // forward steps the backward sweep recomputes
};

class BatchEngine;

class Problem {
    friend class BatchEngine;

public:
    ~Problem();
    fkadj_status init(const fkadj_params& p, double dt, int nt, const int* active_index, int nrows,
                      int ncols, int n_num, const double* gh_num, const double* gamma, int64_t S_ncol,
                      const int64_t* S_colptr, const int64_t* S_rowidx, const double* S_val, double alpha,
                      const fkadj_options* opt, bool need_objective);

    fkadj_status forward(const double* Et, const double* y_ini, int nstep, int ns, double* ys, double* yf) {
        return with_sweeps([&] { return forward_call(Et, y_ini, nstep, ns, ys, yf); });
    }
    fkadj_status objective(const double* Et, const double* y_ini, double* L0, double* LE, double* Lcost,
                           double* yf) {
        return with_sweeps([&] { return objective_call(Et, y_ini, L0, LE, Lcost, yf); });
    }
    fkadj_status grad(const double* Et, const double* y_ini, double* L0, double* LE, double* Lcost,
                      double* gradE, double* yf) {
        return with_sweeps([&] { return grad_call(Et, y_ini, L0, LE, Lcost, gradE, yf); });
    }

    fkadj_status forward_call(const double* Et, const double* y_ini, int nstep, int ns, double* ys, double* yf);
    fkadj_status objective_call(const double* Et, const double* y_ini, double* L0, double* LE, double* Lcost,
                                double* yf);
    fkadj_status grad_call(const double* Et, const double* y_ini, double* L0, double* LE, double* Lcost,
                      double* gradE, double* yf);

    int64_t device_bytes() const;
    // The part of estimate_bytes that refuses no request: small tables, and
    // what the window of z.gh partials on row segments takes beyond all rows on
    // the 16x16 lattice.
    static int64_t estimate_slack(int nrows, int ncols, int nt, int n_num, int grad_mode, int policy, bool want_grad);
    // Bytes of one state of a grid as it lies on the device (3 padded planes).
    static int64_t padded_state_bytes(int nrows, int ncols);
    // Device bytes a problem of this size will hold once a job has run
    // (geometry, work states, adjoint work, Jacobian caches, trajectory store
    // under `policy`), for admission control before anything is allocated.
    // With `sweeps`, what a problem whose steps are sweeps holds (fk_run.h).  A
    // FULL store without k1 kept beside the states (TrajPlan::keep_f).
    static int64_t estimate_bytes(int nrows, int ncols, int nt, int n_num, int64_t nnz, int grad_mode,
                                  int policy, bool want_grad, bool sweeps = false);
    Timing last_timing() const { return timing_; }
    // trajectory plan of the last gradient (policy FULL/SQRT/BINOMIAL, 0 = none yet)
    const TrajPlan& last_plan() const { return traj_plan_; }
    bool has_trajectory() const { return traj_.p != nullptr; }
    int64_t last_launches() const { return launches_; }

    // Sampled per-kernel device times (CUDA events around every k-th launch
    // of each kernel kind; off by default).
    enum Kernel { K_FWD = 0, K_MID = 1, K_ADJ = 2, K_COUNT = 3 };
    void set_profiling(bool on) { profiling_ = on; }
    void kernel_time(int k, double* avg_ms, int64_t* samples) const;
    const DevGrid& grid() const { return g_; }
    int nt() const { return nt_; }
    int n_num() const { return n_num_; }
    cudaStream_t stream() const { return st_; }
    // tile preset per kernel kind; chosen by autotune() unless fixed by options
    enum TileKind { T_FWD = 0, T_MID = 1, T_ADJ = 2, T_EXACT = 3 };
    // reference-mode backward step: k_adj_mid + k_adj_step, or k_adj_fused
    // reading the cached J_F(y_i)^T, or k_adj_fused evaluating it
    enum AdjPath { ADJ_SPLIT = 0, ADJ_FUSED = 1, ADJ_FUSED_RECOMPUTE = 2 };
    int adjoint_path() const { return adj_path_; }
    int fused_tile() const { return tkf_; }
    // A batch engine's problem: stream-ordered device memory from `pool`; with
    // `sweeps`, sweeps whatever its fixed tile (call before init).
    void use_pool(cudaMemPool_t pool, bool sweeps) {
        pool_ = pool;
        shared_ = true;
        own_sweeps_ = sweeps;
    }
    // The preset kernels, which need less device memory (call before init).
    void no_sweeps() { own_sweeps_ = false; }
    // A problem of a one-shot entry point (call before init): device memory
    // from `pool` (null: cudaMalloc), pinned staging from the process's cache.
    void set_oneshot(cudaMemPool_t pool) {
        pool_ = pool;
        oneshot_ = true;
    }
    int tile(int kind) const { return tk_[kind]; }
    void set_tile(int kind, int t) { tk_[kind] = t; }
    // rows per tile in use for a kernel kind (the preset's height, or fewer
    // when the autotuner found a one-wave split faster)
    // rows per tile of a kernel kind as launched (the adjoint step takes its
    // rows on the row-segment lattice only)
    int tile_rows(int kind) const {
        return ty_[kind] > 0 && (kind != T_ADJ || segs_) ? ty_[kind] : tile_shape(tk_[kind]).ty;
    }
    // columns, rows and threads of a kind's tiles as launched
    void launched_tile(int kind, int tile[3]) const {
        if (sweeping()) return run_tile(g_, run_, sms_, kind == T_MID, tile);
        const TileShape t = tile_shape(tk_[kind]);
        tile[0] = t.tx, tile[1] = tile_rows(kind), tile[2] = t.nt;
    }
    // Times every tile preset of every kernel kind on the current initial
    // state (a few launches each) and keeps the fastest per kind.  Results do
    // not depend on the choice (fixed-order reductions).
    fkadj_status autotune();
    fkadj_status autotune_trials();

    // Lower-level pieces (used by the batch / serving layers and the tests).
    // upload_state with y_ini == nullptr re-uses the initial state of the
    // previous call (kept resident on the device).
    fkadj_status upload_state(const double* y_ini, double* d_state);
    // Spline samples of Et on the host; with upload, also the device tables the
    // standalone kernels read (the batched kernels take E by value).
    fkadj_status prepare_E(const double* Et, bool upload = true);
    fkadj_status step_forward(int i, const double* yin, double* yout, double* k1 = nullptr);
    // n forward steps from step i, src -> last; of the states between, those
    // after `first` steps and every `every` more go to out, out +
    // state_elems(), ... when out is non-null; `keep` receives per step k1 = f
    // of the state before it (reference mode: per-step launches) or the three
    // stage states (exact mode: sweeps).  One launch where the grid is swept
    // (sweeping()), n launches otherwise.
    fkadj_status sweep_forward(int i, int n, const double* src, double* last, double* out = nullptr,
                               double* keep = nullptr, int first = 1, int every = 1);
    // The same as a job of a launch (its exchange tags are taken: launch jobs
    // in the order they were made).
    FwdJob forward_job(int i, int n, const double* src, double* last, double* out, double* keep, int first, int every);
    struct AdjointChunk {
        int n;        // steps
        bool replay;  // the points come from a forward sweep of the same steps into pts_
        MidJob mid;   // ... or from this (reference mode)
        AdjJob adj;   // its exchange tags are still to be taken (take_tags)
    };
    AdjointChunk adjoint_chunk(int top, int hi, int lo, const double* y_hi, const double* mid, const double* y_lo,
                               const double* stages, const double* z, double* z2, int most);
    void take_tags(AdjointChunk& c) {
        c.adj.r.epoch = epoch_;
        epoch_ += (unsigned long long)c.n;
    }
    // Backward steps hi .. lo + 1 of a swept problem, z -> z (the pair is
    // swapped as it goes): y_hi, y_lo the states at both ends, mid the states
    // lo + 1 .. hi - 1 in a row, stages (exact mode; null: replayed) the stage
    // states of steps lo .. hi - 1 in a row.  replayed: where a replay leaves
    // the states between (mid, where they are not there yet).
    fkadj_status sweep_adjoint(int hi, int lo, const double* y_hi, const double* mid, const double* y_lo,
                               const double* stages, double*& z, double*& z2, double* replayed = nullptr);
    fkadj_status init_sweeps(const uint8_t* flags);
    fkadj_status ensure_exchange();
    // Sweeps as launches of the tile kernels from here on (the same bits): the
    // device refused a cooperative launch of the grid's tiles, a CTA per SM (a
    // stream may see fewer SMs than the device has).
    void no_run() {
        no_coop_ = false;
        run_ = RunShape();
        xchg_.release();
    }
    // What only sweeps use.  (Kept stage states go with the plan: ensure_traj.)
    void drop_sweep_buffers() {
        for (DevBuf* b : {&xchg_, &pts_}) b->release();
    }
    // whether this problem's steps are sweeps (fk_run.h): one launch each where
    // run_.id >= 0, the tile kernels otherwise
    bool sweeping() const { return swept_ && !run_off_; }
    double* state_buf(int k) const { return work_.as<double>() + (size_t)k * state_elems(); }
    size_t state_elems() const { return (size_t)3 * g_.plane; }
    size_t state_bytes() const { return state_elems() * sizeof(double); }

private:
    fkadj_status fail_cuda(cudaError_t e, const char* what);
    // brackets a launch of kernel kind k with sampled events when profiling
    cudaError_t prof_begin(int k, int steps = 1);
    cudaError_t prof_end(int k);
    fkadj_status prof_collect();
    // FKADJ_ERR_TIMEOUT when a kernel's bounded wait expired since the last check
    fkadj_status check_fault();
    // a call that sweeps, repeated with per-step launches where check_fault found FAULT_NAN
    template <class Call> fkadj_status with_sweeps(Call&& call);
    // Resolves the checkpoint policy.  AUTO takes FULL when the budget holds
    // every state, else whichever of SQRT and BINOMIAL fits and costs less,
    // counted in forward-step equivalents (the work of each per backward step
    // included); with sqrt_or_full_only (the batch
    // engine, which runs no binomial schedule) BINOMIAL only when SQRT does not
    // fit.
    double binomial_step_cost(double* forward_us) const;
    fkadj_status default_budget();
    fkadj_status plan_trajectory(TrajPlan& tp, bool sqrt_or_full_only = false);
    int64_t kept_states(const TrajPlan& tp) const;
    fkadj_status ensure_traj(const TrajPlan& tp);
    fkadj_status run_objective(const double* yT, double* L0);
    fkadj_status objective_async(const double* yT);
    fkadj_status grad_exact_backward(const TrajPlan& tp, double* lam, double* lam2);
    fkadj_status advance(int a, int m, const double* src, double* dst);
    fkadj_status reverse_binomial(int nt, double* y0, std::vector<double*>& free,
                                  const std::function<fkadj_status(int, int, const double*, const double*)>& visit);
    // all_rows: keep the z.gh partials of every step (the batch engine);
    // otherwise a window of kPartialWindow rows reduced as the sweep goes.
    fkadj_status ensure_adjoint_work(bool all_rows = false);
    // z.gh partial row `row` of group g (exact mode: 3 groups of nt rows;
    // reference mode: one group of nt+1 rows) in the window
    double* prow(int g, int row) const {
        return partial_.as<double>() + ((size_t)g * pwin_ + (size_t)(row % pwin_)) * nsb_;
    }
    int groups() const { return grad_mode_ == FKADJ_GRAD_EXACT ? 3 : 1; }
    // Adds to l, per group of partial sums, the reduction into zgh of the
    // window of rows from `row` on (clipped to the group's rows), or of rows
    // row0 .. row0+n-1; the latter must not wrap around the window (a sqrt
    // segment's rows, with the window a whole number of segments).
    void sum_window(SumList& l, int row) const;
    void sum_range(SumList& l, int row0, int n) const;
    cudaError_t flush_rows(int row);
    cudaError_t flush_range(int row0, int n);
    static constexpr int kPartialWindow = 512;
    static int partial_window(int nt, bool exact, int stride, size_t nsb16, size_t nsbseg, bool segs);
    fkadj_status download_grid(const double* d_state, double* host_dense);
    double* slot(int k) const { return traj_.as<double>() + (size_t)k * state_elems(); }
    double* segslot(int k) const { return seg_.as<double>() + (size_t)k * state_elems(); }
    double* fslot(int k) const { return kf_.as<double>() + (size_t)k * state_elems(); }
    // E samples of step i read from the device tables (uploaded by prepare_E)
    const double* etab() const { return Ed_.as<double>(); }
    EStep efwd(int i) const {
        const double* t = etab();
        return EStep::table(t + i, t + (nt_ + 1) + i, t + i + 1);  // Et[i], E(t_i + dt/2), Et[i+1]
    }
    EStep emid(int i) const {
        const double* t = etab();
        return EStep::table(t + i - 1, t + i, t + (2 * nt_ + 1) + i - 1);  // Et[i-1], Et[i], E(t_{i-1} + dt/3)
    }
    // The gradient's device work after the initial state is in place: forward
    // sweep, objective, backward sweep, reductions, and the copies of L0 and the
    // z.gh rows into pinned host memory.  Issued directly or captured once into a
    // CUDA graph and replayed (use_graph).
    fkadj_status grad_sequence(const TrajPlan& tp, bool exact, double** yT);
    fkadj_status grad_replay(const TrajPlan& tp, bool exact, double** yT);
    // segment graphs of a gradient run as plain launches (fk_engine.cu)
    bool segment_graphs_wanted() const;
    fkadj_status segment_begin();
    fkadj_status segment_launch();
    void segment_abort();
    void drop_segment_graphs();
    cudaGraphExec_t seg_exec_[2] = {nullptr, nullptr};
    cudaEvent_t seg_done_[2] = {nullptr, nullptr};
    int seg_next_ = 0;
    bool seg_on_ = false;
    void drop_graph();

    fkadj_params p_{};
    DevModel P_{};
    DevGrid g_{};
    HermiteW hw_{};
    double dt_ = 0, alpha_ = 0, gamma_[3] = {0, 0, 0};
    int nt_ = 0, n_num_ = 0, device_ = 0, nsbx_ = 0, nsby_ = 0, nsb_ = 0;
    // z.gh partials on the row-segment lattice (nsb_ = nsbx_ x nrows; the
    // adjoint step's tiles then take balanced rows) instead of the 16x16 one
    // (nsb_ = nsbx_ x nsby_); chosen by ensure_adjoint_work
    bool segs_ = false;
    int tk_[4] = {0, 0, 0, 0};  // tile preset per kernel kind (TileKind)
    int tkf_ = 0;               // fused reference-adjoint preset (fused_shape)
    int adj_path_ = 0;          // AdjPath of the reference-mode backward step
    int forced_path_ = -1;      // AdjPath fixed by FKADJ_ADJ_PATH (-1: autotuned)
    // Jacobian caches of the split backward step (FKADJ_JCACHE): 2 = J(yh)
    // from the midpoint kernel and J(y_{i-1}) carried to the next step; 1 =
    // the carry only, the step evaluates J(yh); 0 = the step evaluates both
    int jcache_mode_ = 2;
    int ty_[4] = {0, 0, 0, 0};  // rows per tile per kind (0 = the preset's height)
    bool autotune_ = true, tuned_ = false, tuned_fwd_ = false;
    bool tiles_fixed_ = false;  // FKADJ_TILES fixed every kind's preset: autotune() keeps them
    bool own_stream_ = false, have_obj_ = false;
    cudaMemPool_t pool_ = nullptr;
    int verbose_ = 0;
    int grad_mode_ = FKADJ_GRAD_REF, ckpt_policy_ = FKADJ_CKPT_AUTO;
    int64_t ckpt_budget_ = 0;
    cudaStream_t st_ = nullptr;
    cudaEvent_t ev_[3] = {nullptr, nullptr, nullptr};

    // device buffers
    DevBuf gh_, wc_, pos_, Srow_, Scol_, Sval_, yc_, zc_, opart_, osum_;
    DevBuf fault_;     // this problem's fault word: set by a step kernel whose bounded wait expired
    unsigned* fault() const { return fault_.as<unsigned>(); }
    DevBuf flags_;     // where the grid is swept: geometry flags per padded cell (CELL_*), the adjoint
                       // sweeps' flags likewise, and per 16-cell row segment whether it holds a source cell
    size_t flag_bytes() const { return ((size_t)g_.plane + 7) / 8 * 8; }
    const uint8_t* adj_flags() const { return flags_.as<uint8_t>() + flag_bytes(); }
    const uint8_t* segment_flags() const { return flags_.as<uint8_t>() + 2 * flag_bytes(); }
    DevBuf xchg_;      // the sweeps' edge exchange
    DevBuf pts_;       // points between the states of one chunk of an adjoint sweep
    int sms_ = 0;
    static int sweep_chunk_of(int64_t state_bytes, bool exact);
    int sweep_chunk() const;
    RunShape run_;     // how the grid is swept in one launch (id -1: it does not fit)
    bool swept_ = false;
    bool zero_holes_ = false;  // what zbuf_ holds at holes
    unsigned long long epoch_ = 0;  // steps swept so far (the exchange's tags)
    // the preset kernels after all: a sweep met a NaN away from the holes
    // (FAULT_NAN), which they contain
    bool run_off_ = false;
    bool nan_seen_ = false;
    bool no_coop_ = false;     // a cooperative launch was refused as too large
    bool refused_ = false;     // the last plan: refused by the caller's budget, whatever memory there is
    bool own_sweeps_ = true;  // false where memory is short
    bool shared_ = false;     // a batch engine's problem
    cudaEvent_t eup_ = nullptr;  // of such a problem: its E tables' upload
    DevBuf work_;      // 4 states: two ping-pong, z pair is separate
    DevBuf zbuf_;      // 2 adjoint states
    DevBuf yh_;        // midpoint state
    DevBuf partial_;   // (nt+1) x ntiles zgh partials
    DevBuf zgh_;       // nt+1
    DevBuf traj_, seg_;
    DevBuf kf_;        // kept k1 = f(y_t) per stored / recomputed state (TrajPlan::keep_f)
    DevBuf y0res_;     // resident initial state
    DevBuf stg_;       // stage states Y2, Y3, Y4 of one step (exact mode)
    DevBuf jcache_;    // cached Jacobians (reference mode): J(y) ping-pong + J(yh)
    DevBuf fcache_;    // f(y) carried between backward steps (reference mode)
    DevBuf Ed_;        // E tables: Et (nt+1), E at half steps (nt), E at third steps (nt)
    double* Ehost_ = nullptr;  // pinned staging of the E tables
    double* hres_ = nullptr;   // pinned results: L0 partial sum, then the z.gh rows
    size_t hres_n_ = 0;
    size_t Ehost_n_ = 0;       // capacity of Ehost_ (doubles)
    bool e_ready_ = false;     // the E tables' buffers are there
    double* setup_ = nullptr;  // pinned block of the set-up's uploads
    size_t setup_n_ = 0;
    double* frame_ = nullptr;  // pinned staging of a downloaded state
    size_t frame_n_ = 0;
    DevBuf dense_;             // a state packed for download
    bool oneshot_ = false;
    bool have_y0_ = false;

    // captured gradient sequence
    struct GraphKey {
        int policy = -1, nslots = 0, seg_slots = 0, keep_f = 0, exact = 0, gen = 0, path = 0, tkf = 0;
        int tk[4] = {0, 0, 0, 0}, ty[4] = {0, 0, 0, 0};
        bool operator==(const GraphKey& o) const;
    };
    bool graphs_ = true;         // FKADJ_NO_GRAPHS=1 in the environment turns replay off
    cudaGraphExec_t gexec_ = nullptr;
    GraphKey gkey_{};
    GraphKey seen_key_{};        // configuration of the previous gradient
    GraphKey graph_key(const TrajPlan& tp, bool exact) const;
    int64_t glaunches_ = 0;
    double* gyT_ = nullptr;
    int buf_gen_ = 0;            // bumped whenever a buffer the sequence uses is reallocated
    int pwin_ = 1;               // rows per group in the z.gh partial window
    bool capturing_ = false;
    TrajPlan traj_plan_{};

    // sampled kernel timing
    bool profiling_ = false;
    int prof_every_ = 1;
    int64_t kcount_[K_COUNT] = {0, 0, 0};
    int64_t ksamples_[K_COUNT] = {0, 0, 0};
    double kms_[K_COUNT] = {0, 0, 0};
    struct ProfRec {
        int k, n;
        cudaEvent_t a, b;
    };
    std::vector<ProfRec> prof_pool_;
    size_t prof_used_ = 0;
    bool prof_open_ = false;

    // host
    std::vector<double> Et_, ypp_, Eh_, E3_;
    NakSpline* spline_ = nullptr;
    Timing timing_{};
    int64_t launches_ = 0;
};

template <class Call>
fkadj_status Problem::with_sweeps(Call&& call) {
    nan_seen_ = refused_ = false;
    fkadj_status s = ensure_exchange();
    if (!s) s = call();
    if (no_coop_) {
        no_run();
        s = call();
    }
    if (s == FKADJ_ERR_NOMEM && sweeping() && !refused_) {
        // the preset kernels need less memory; where they lack it too, sweeps
        // were not what it was short for
        drop_sweep_buffers();
        swept_ = false;
        s = call();
        if (s == FKADJ_ERR_NOMEM) swept_ = true;
        return s;
    }
    if (!nan_seen_) return s;
    // once more with the preset kernels.  A one-shot problem (the server's)
    // never holds both paths' buffers; a resident one gives the sweeps' up
    // only where the device lacks the memory (the next call sweeps again)
    run_off_ = true;
    if (oneshot_) drop_sweep_buffers();
    s = call();
    if (s == FKADJ_ERR_NOMEM && !refused_ && (xchg_.p || pts_.p)) {
        drop_sweep_buffers();
        s = call();
    }
    run_off_ = false;
    return s;
}

// The binomial schedule's first chain of checkpoints (the states the forward
// sweep stores), and the forward steps its reversal then recomputes.
std::vector<int> binomial_spine(int nt, int free_slots);
int64_t binomial_recompute_steps(int nt, int free_slots);

// Memory the one-shot entry points keep between calls: the per-device pool
// (null when FKADJ_ONESHOT_POOL=0) and its release (fkadj_release_cached_memory).
cudaMemPool_t oneshot_pool(const fkadj_options* opt);
fkadj_status release_oneshot_memory();

}  // namespace fkadj
