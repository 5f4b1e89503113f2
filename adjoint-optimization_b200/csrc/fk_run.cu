// fk_run.cu -- time sweeps as one launch each (sm_100a).
//
// A per-step launch of the forward step at 512 x 512 takes 15.2 us in a
// replayed graph, of which about 4 us are the launch boundary and the tile
// loads, and the rest runs the FP64 pipe half busy.  Where the grid's tiles
// fit the device at once (one CTA per SM), a whole sweep runs as one
// cooperative launch instead (11.0 us a step): each CTA keeps its tile in shared memory from
// step to step and exchanges only the 4-cell edges with its eight neighbours
// through L2, waiting for its own neighbours and no one else.
//
// The exchange carries its own arrival: every edge value travels as one
// 16-byte store of the value and the step's number, and the reader polls the
// value it needs until the number is right.  A flag per tile instead (stores,
// barrier, fence, flag; poll, barrier, loads) measured 5 us a step: the fence
// and the flag are round trips of their own.
//
// Inside a step, what bounds the work is the FP64 pipe (80 instructions per
// evaluation, 2 cycles each per scheduler) and then the shared-memory data
// path; so
//  - a thread owns R rows of one column and walks down them, keeping the
//    column's three values in registers: per field and cell the stencil reads
//    (R + 2 + 2 R) / R values instead of 5;
//  - the RK accumulator lives in registers (the owner never changes) and the
//    step-start state stays in its own window, so no stage reads global memory;
//  - missing neighbours come from per-cell flags, six bits per row held in one
//    register for the whole sweep, as selects: the NaN test with its branch,
//    taken by one warp in five, cost 2.4 us a step at 512 x 512, a separate
//    pass over the flagged cells 1.5-2 us.
#include "fk_run.h"

#include <algorithm>
#include <type_traits>
#include <utility>
#include <vector>

#include "fk_bulk.cuh"
#include "fk_ring.cuh"

namespace fkadj {

namespace {

// Kernel instances (id, TX, R, TYM): tiles of TX columns and up to TYM rows;
// TYM + 6 is a multiple of R (the first stage's region, TYM + 6 rows of it).
// A grid takes the one of least cost among those whose tiles fit the device
// (ShapeInfo::cost), and so do a batch's launches.  Forward and backward us a
// step with each (a dash: does not fit):
//             64x5x29    64x4x22   64x3x15   32x3x30   32x2x18   16x2x34   16x1x14
//   128x128   6.5 13.5   6.0 11.0  5.0 8.1   4.3 7.0   3.5 5.8   3.7 6.1   3.0 4.6
//   256x256   7.6 15.3   6.3 12.0  5.8 9.5   5.6 9.3   5.4 8.5   5.7 9.0      -
//   320x320   8.3 16.8   7.2 13.2  7.0 11.0  6.8 10.9     -         -         -
//   384x384   8.8 17.0   8.2 14.2     -         -         -         -         -
//   437x501  11.0 19.2      -         -         -         -         -         -
// (32x4x42, not listed, is level with 64x4x22 at 384x384: 8.3 14.1.)
#define FKADJ_RUN_LIST(X) \
    X(0, 64, 5, 29)       \
    X(1, 64, 3, 15)       \
    X(2, 32, 3, 30)       \
    X(3, 32, 2, 18)       \
    X(4, 16, 2, 34)       \
    X(5, 16, 1, 14)       \
    X(6, 64, 4, 22)       \
    X(7, 32, 4, 42)

template <int TX_, int R_, int TYM_>
struct Shape {
    static constexpr int TX = TX_, R = R_, TYM = TYM_;
    static constexpr bool RESIDENT = true;  // the tile stays in window A from step to step
    static constexpr int RW = TX + 2 * HALO;  // window width = pitch of every buffer
    // Buffers, three planes each, all addressed in window coordinates (row 0 =
    // 4 rows above the tile): A, the step-start state, rows 0 .. TYM + 7; B,
    // rows 1 .. TYM + 6; C, rows 2 .. TYM + 5; then one plane G of the source,
    // rows 1 .. TYM + 6.  A thread's column may read two rows past C's last
    // plane (for rows it does not keep): they lie in G.  Last, the ring's table
    // (ring_table).
    static constexpr int PA = (TYM + 8) * RW, PB = (TYM + 6) * RW, PC = (TYM + 4) * RW;
    static constexpr int THREADS = ((RW * ((TYM + 6) / R) + 31) / 32) * 32;
    static constexpr int RING = 8 * RW + 8 * TYM;  // cells around the largest tile
    static constexpr size_t SMEM = sizeof(double) * (size_t)(3 * (PA + PB + PC) + PB) + RING * sizeof(int2);
    static constexpr size_t SMEM_EXACT = SMEM + sizeof(double) * (size_t)PB;  // and one more plane
    static_assert((TYM + 6) % R == 0, "the first stage's rows are whole columns of R");
    static_assert(R <= 5, "six flag bits a row in one register");
    static_assert(SMEM_EXACT + 768 <= 232448, "one CTA's shared memory");
    static_assert(THREADS <= 512, "128 registers per thread");
};

// Tiles of the per-step kernels of larger grids (k_fwd_tile, k_adj_tile): the
// same stages, with a second window A that takes the next tile's while this
// one computes, the source read from global memory, and the terms of the z.gh
// sums in planes of their own (three in the exact mode).
struct TileShapeBig {
    static constexpr int TX = 64, R = 4, TYM = 22;
    static constexpr bool RESIDENT = false;
    static constexpr int RW = TX + 2 * HALO;
    static constexpr int PA = (TYM + 8) * RW, PB = (TYM + 6) * RW, PC = (TYM + 4) * RW, TERM = TYM * TX;
    static constexpr int THREADS = ((RW * ((TYM + 6) / R) + 31) / 32) * 32;
    static constexpr size_t SMEM = sizeof(double) * (size_t)(3 * (2 * PA + PB + PC) + 3 * TERM);
    static_assert((TYM + 6) % R == 0 && THREADS <= 512 && SMEM + 256 <= 232448, "one CTA per SM");
    static_assert(3 * TERM >= 2 * RW, "reads past C stay in the allocation");
};

// The jobs of a launch, in the order of their tiles.  A kernel of several
// copies its CTA's job to shared memory first (take): indexed where they lie,
// among the parameters, one instance ended in an illegal instruction.
constexpr int kRunJobs = 16;
template <class Job>
struct RunJobs {
    int n;
    Job job[kRunJobs];
    // *j <- the job of a tile; ends with the CTA synchronised
    __device__ __forceinline__ void take(int tile, Job* j) const {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int q = 0; q < kRunJobs; ++q)
                if (q < n && tile >= job[q].tile0 && (q + 1 >= n || tile < job[min(q + 1, kRunJobs - 1)].tile0)) *j = job[q];
        }
        __syncthreads();
    }
};

// What a thread knows of its column (constant over the sweep).
struct Column {
    int c, r0;      // window column, first window row
    int o;          // offset of (r0, c) from the window's origin in a state plane
    unsigned bits;  // CELL_* of row r0 + k at bit 6 k
};

// One forward stage on the tile grown by E cells, for the thread's own cells:
// k = f(src), then
//   MODE 0: dst = y0 + cY k, D  = cD k     (first stage: src is y0's window)
//   MODE 1: dst = y0 + cY k, D += cD k     (middle stages)
//   MODE 2: y0 <- (y0 + D) + cD k          (last stage)
// with y0 in window A; the result of the tile's own cells also to `out` (null:
// nowhere) and, in the last stage, the tile's edges to the exchange x (null:
// nowhere).  A hole's own value is NaN in A and so in every result
// that leaves the tile; what B and C hold there is never read as a neighbour.
template <int E, class S, int MODE, int PS, int PT>
__device__ __forceinline__ void fwd_rows(const DevModel& P, const Column& T, const double* src, double* dst, double* A,
                                         const double* G, double (&D)[S::R][3], int rows, int ld, long long plane,
                                         double Ev, double cY, double cD, double* __restrict__ out,
                                         Tagged* __restrict__ x, unsigned long long tag, bool& bad) {
    constexpr int RW = S::RW;
    if (T.c < HALO - E || T.c >= HALO + S::TX + E) return;
    const int q0 = T.r0 * RW + T.c;
    const double* Y = src + q0;
    // opaque: what follows from the flags is the same at every step, and the
    // compiler would keep it in registers (and spill) from step to step
    unsigned bits = T.bits;
    asm volatile("" : "+r"(bits));
    double n[3], m[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) n[f] = Y[f * PS - RW], m[f] = Y[f * PS];
#pragma unroll
    for (int k = 0; k < S::R; ++k) {
        const int r = T.r0 + k;
        const unsigned b = bits >> (6 * k);
        // a missing neighbour is read where the opposite one is; the value
        // below then stands in for a hole's, which no one uses
        const double* ps = Y + ((b & CELL_S) ? k - 1 : k + 1) * RW;
        const double* pw = Y + k * RW + ((b & CELL_W) ? 1 : -1);
        const double* pe = Y + k * RW + ((b & CELL_E) ? -1 : 1);
        double s[3];
        double gv = 0.0;
        if (b & CELL_SOURCE) gv = S::RESIDENT ? G[q0 + k * RW] : __ldg(G + T.o + k * ld);
#pragma unroll
        for (int f = 0; f < 3; ++f) s[f] = ps[f * PS];
        if (r >= HALO - E && r < HALO + rows + E) {
            double t[3], kk[3];
#pragma unroll
            for (int f = 0; f < 3; ++f) t[f] = lap4((b & CELL_N) ? s[f] : n[f], s[f], pw[f * PS], pe[f * PS], m[f]);
            fk_field(P, m, t, Ev, gv, kk[0], kk[1], kk[2]);
            double* a = A + q0 + k * RW;
            if (MODE == 2) {
                double o[3];
#pragma unroll
                for (int f = 0; f < 3; ++f) o[f] = fma(cD, kk[f], a[f * S::PA] + D[k][f]);
                if (S::RESIDENT) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) a[f * S::PA] = o[f];
                }
                bad = bad || (isnan(o[0]) && (b & CELL_ACTIVE));
                if (out) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) out[f * plane + T.o + k * ld] = o[f];
                }
                if (x && (r < 2 * HALO || r >= rows || T.c < 2 * HALO || T.c >= S::TX)) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) put_tagged(x + f * plane + T.o + k * ld, o[f], tag);
                }
            } else {
                double o[3];
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const double y0 = MODE == 0 ? m[f] : a[f * S::PA];
                    dst[f * PT + q0 + k * RW] = o[f] = fma(cY, kk[f], y0);
                    D[k][f] = MODE == 0 ? cD * kk[f] : fma(cD, kk[f], D[k][f]);
                }
                if (out && r >= HALO && r < HALO + rows && T.c >= HALO && T.c < HALO + S::TX) {
#pragma unroll
                    for (int f = 0; f < 3; ++f)
                        out[f * plane + T.o + k * ld] = (b & CELL_ACTIVE) ? o[f] : __longlong_as_double(-1);
                }
            }
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) n[f] = m[f], m[f] = s[f];
    }
}

// A sweep of r.n forward steps (launch_fwd_run: cooperative, one CTA per
// tile).  The exchange area is two 3-plane grids of Tagged, used in turn: a
// tile writes step k + 2's edges over step k's only after it has read its
// neighbours' step k + 1, which they published after they had read step k.
template <class S>
__device__ __forceinline__ void fwd_run(const DevModel& P, const FwdJob& J) {
    constexpr int TX = S::TX, R = S::R;
    const DevGrid& g = J.g;
    const FwdRun& r = J.r;
    const double* __restrict__ gh = J.gh;
    const uint8_t* __restrict__ cells = J.cells;
    const int ty = J.ty;
    constexpr int RW = S::RW;
    extern __shared__ double4 smem_raw[];
    __shared__ uint64_t bar;
    double* A = reinterpret_cast<double*>(smem_raw);
    double* B = A + 3 * S::PA - RW;
    double* C = A + 3 * (S::PA + S::PB) - 2 * RW;
    double* G = A + 3 * (S::PA + S::PB + S::PC) - RW;
    const int tile = blockIdx.x - J.tile0, by = tile / J.ntx, bx = tile - by * J.ntx;
    const int i0 = by * ty, j0 = bx * TX;
    const int rows = min(ty, g.nrows - i0);
    const long long off = (long long)i0 * g.ld + j0;  // window origin: logical (i0 - 4, j0 - 4)

    int2* ring = reinterpret_cast<int2*>(G + RW + S::PB);
    const int nring = ring_table<S>(ring, g.ld, rows, i0, j0, g.nrows, J.ntx * TX);
    exp_table_init();
    const uint32_t b = bulk_begin(&bar);
    __syncthreads();
    bulk_arrive(b, bulk_bytes<RW>(rows + 2 * HALO));
    __syncthreads();
    {
        const int nr = rows + 2 * HALO;
        for (int t = threadIdx.x; t < 3 * nr; t += blockDim.x) {
            const int f = t / nr, row = t - f * nr;
            bulk_row<RW>(b, A + f * S::PA + row * RW, r.src + off + f * g.plane + (long long)row * g.ld);
        }
    }
    Column T;
    {
        const int col = threadIdx.x / RW;
        T.c = threadIdx.x - col * RW;
        T.r0 = 1 + col * R;
        T.o = T.r0 * g.ld + T.c;
        T.bits = 0;
        if (T.r0 >= rows + 7) T.c = -1;  // no rows: out of every stage's columns
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (T.c >= 1 && T.c < TX + 7 && T.r0 + k < rows + 7) {
                const unsigned f = cells[off + T.o + k * g.ld];
                T.bits |= f << (6 * k);
                G[(T.r0 + k) * RW + T.c] = gh[off + T.o + k * g.ld];
            }
        }
    }
    if (!bulk_wait_cta(b, r.fault)) return;
    __syncthreads();
    double D[R][3];
    bool bad = false;
    for (int k = 0; k < r.n; ++k) {
        // what a stage needs is worked out where it starts: registers are short
        auto stage_out = [&](int st) { return r.stages ? r.stages + (3LL * k + st) * r.stride + off : nullptr; };
        fwd_rows<3, S, 0, S::PA, S::PB>(P, T, A, B, A, G, D, rows, g.ld, g.plane, __ldg(r.Et + k), 0.5 * P.dt,
                                        1.0 / 6.0 * P.dt, stage_out(0), nullptr, 0, bad);
        __syncthreads();
        fwd_rows<2, S, 1, S::PB, S::PC>(P, T, B, C, A, G, D, rows, g.ld, g.plane, __ldg(r.Eh + k), 0.5 * P.dt,
                                        1.0 / 3.0 * P.dt, stage_out(1), nullptr, 0, bad);
        __syncthreads();
        fwd_rows<1, S, 1, S::PC, S::PB>(P, T, C, B, A, G, D, rows, g.ld, g.plane, __ldg(r.Eh + k), P.dt,
                                        1.0 / 3.0 * P.dt, stage_out(2), nullptr, 0, bad);
        __syncthreads();
        const bool end = k == r.n - 1;
        const unsigned long long tag = r.epoch + k + 1;
        Tagged* x = static_cast<Tagged*>(r.exchange) + (tag & 1) * (3 * g.plane) + off;
        {
            double* out = end ? r.last : nullptr;
            if (!end && r.out && k + 1 >= r.first) {
                const int m = (k + 1 - r.first) / r.every;
                if (m * r.every == k + 1 - r.first) out = r.out + m * r.stride;
            }
            fwd_rows<0, S, 2, S::PB, S::PB>(P, T, B, nullptr, A, G, D, rows, g.ld, g.plane, __ldg(r.Et + k + 1), 0.0,
                                            P.dt_6, out ? out + off : nullptr, end ? nullptr : x, tag, bad);
        }
        if (end) break;
        if (!read_ring<S>(A, ring, nring, x, tag, g.plane, r.fault)) return;
    }
    // A NaN in an active cell came from the inputs or from a state that blew
    // up: the per-step kernels contain it (their stencil takes any NaN
    // neighbour for missing), this sweep lets it spread.  The host repeats the
    // call with them.
    if (bad) atomicOr(r.fault, FAULT_NAN);
}

template <int TX, int R, int TYM>
__global__ void __launch_bounds__(Shape<TX, R, TYM>::THREADS, 1) k_fwd_run(const DevModel P, const FwdJob j) {
    fwd_run<Shape<TX, R, TYM>>(P, j);
}

template <int TX, int R, int TYM>
__global__ void __launch_bounds__(Shape<TX, R, TYM>::THREADS, 1)
    k_fwd_jobs(const DevModel P, const RunJobs<FwdJob> jobs) {
    __shared__ FwdJob j;
    jobs.take(blockIdx.x, &j);
    fwd_run<Shape<TX, R, TYM>>(P, j);
}

// ------------------------------------------------------------ adjoint sweeps
//
// A backward step of either mode is four stages k_s = L^T a_s + J_F(Y_s)^T a_s
// of the same shape: stage s on the tile grown by 4 - s cells, each at its own
// state Y_s, which no stage changes (the reference mode: y_i, the midpoint
// twice, y_{i-1}; the exact mode: the step's stage states Y4, Y3, Y2 and y_s).
// The sweep therefore is k_fwd_run's with the Jacobian evaluated at a state
// read from global memory, one row ahead of its use.  Evaluating J on the
// halo again (4.6 times a cell and step) costs 490 FP64 instructions a cell;
// the per-step kernels read the seven entries cached by other kernels
// instead, 250 B a cell and step through L2.  At 512 x 512 a step takes 19.8
// us, 20 with the caches, but the kernel that made them (14 us a step) is now
// k_mid_run (6.6 us); at 256 x 256 8.6 us, at 128 x 128 4.6.  Of the 19.8 us
// the FP64 pipe is busy 42 %; 16 warps wait on fixed latencies, the points'
// loads, the exchange and the barriers.  (Keeping J(yh) of the second stage
// for the third, through an L2 scratch, took 17 % of the FP64 instructions
// away and 1 % of the time: the 286 KB a step cost the SM's port as much.)
//
// Holes and everything off the grid hold 0 here, in the buffers and in z's
// states: a missing neighbour then adds nothing to the plain sum, and only the
// neighbours that mirrored this cell are added once more.

// Row k of a column's values of state y (its window's origin), 0 past the tile
template <class S>
__device__ __forceinline__ void load_point(const Column& T, int k, int rows, int ld, long long plane,
                                           const double* __restrict__ y, double (&v)[3]) {
    const bool on = T.c >= 1 && T.c < S::TX + 7 && T.r0 + k < rows + 7;
#pragma unroll
    for (int f = 0; f < 3; ++f) v[f] = on ? __ldg(y + f * plane + T.o + k * ld) : 0.0;
}

// A cell's term of a z.gh sum: NaN counts as 0, as does a cell without source
__device__ __forceinline__ double source_term(unsigned b, double z, double gh) {
    const double t = z * gh;
    return (b & CELL_SOURCE) && !isnan(t) ? t : 0.0;
}

// One backward stage on the tile grown by E cells, for the thread's own cells:
// k = L^T src + J_F(y)^T src, then in the reference mode
//   MODE 0: dst = z0 + cA k, D  = cB k
//   MODE 1: dst = z0 + cA k, D += cB k
//   MODE 2: z0 <- (z0 + D) + cB k
// and in the exact mode, where src is z0 = lambda itself in the first stage
// and k there is scaled by cS = dt/6 (a_4 = dt/6 lambda),
//   MODE 0: dst = cB z0 + cA k, D  = k;  MODE 1: the same, D += k
//   MODE 2: z0 <- z0 + (D + k)
// with z0 in window A.  yv holds the first row of y.  keep: in a resident
// tile's exact mode, where the first stage leaves a_3 on u; else the planes of
// the z.gh sums' terms (gh: the source's window origin).
template <int E, class S, int MODE, int PS, int PT, bool EXACT>
__device__ __forceinline__ void adj_rows(const DevModel& P, const Column& T, const double* src, double* dst, double* A,
                                         double (&D)[S::R][3], double (&yv)[3], const double* __restrict__ y, int rows,
                                         int ld, long long plane, double cA, double cB, double cS, double* keep,
                                         const double* __restrict__ gh, double* __restrict__ out, Tagged* __restrict__ x, unsigned long long tag) {
    constexpr int RW = S::RW;
    if (T.c < HALO - E || T.c >= HALO + S::TX + E) return;
    const int q0 = T.r0 * RW + T.c;
    const double* Z = src + q0;
    unsigned bits = T.bits;
    asm volatile("" : "+r"(bits));  // as in fwd_rows
    double n[3], m[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) n[f] = Z[f * PS - RW], m[f] = Z[f * PS];
#pragma unroll
    for (int k = 0; k < S::R; ++k) {
        const int r = T.r0 + k;
        const unsigned b = bits >> (6 * k);
        double s[3], yn[3];
        if (k + 1 < S::R) load_point<S>(T, k + 1, rows, ld, plane, y, yn);
        double gv = 0.0;
        if (!S::RESIDENT && (MODE == 2 || EXACT) && (b & CELL_SOURCE)) gv = __ldg(gh + T.o + k * ld);
#pragma unroll
        for (int f = 0; f < 3; ++f) s[f] = Z[f * PS + (k + 1) * RW];
        if (r >= HALO - E && r < HALO + rows + E) {
            double t[3], kk[3];
#pragma unroll
            for (int f = 0; f < 3; ++f)
                t[f] = lap4(n[f], s[f], Z[f * PS + k * RW - 1], Z[f * PS + k * RW + 1], m[f]);
            if (b & (CELL_2N | CELL_2S | CELL_2W | CELL_2E)) {
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    if (b & CELL_2N) t[f] += n[f];
                    if (b & CELL_2S) t[f] += s[f];
                    if (b & CELL_2W) t[f] += Z[f * PS + k * RW - 1];
                    if (b & CELL_2E) t[f] += Z[f * PS + k * RW + 1];
                }
            }
            const JacT J = fk_jacT(P, yv[0], yv[1], yv[2]);
            adj_field(P, J, m, t, kk[0], kk[1], kk[2]);
            const bool act = b & CELL_ACTIVE_ADJ;
            double* a = A + q0 + k * RW;
            const int term = (r - HALO) * S::TX + T.c - HALO;
            if (MODE == 2) {
                double o[3];
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    o[f] = EXACT ? a[f * S::PA] + (D[k][f] + kk[f]) : fma(cB, kk[f], a[f * S::PA] + D[k][f]);
                if (S::RESIDENT && act) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) a[f * S::PA] = o[f];
                }
                if constexpr (!S::RESIDENT && !EXACT) keep[term] = source_term(b, o[0], gv);
                if (out) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) out[f * plane + T.o + k * ld] = act ? o[f] : 0.0;
                }
                if (x && (r < 2 * HALO || r >= rows || T.c < 2 * HALO || T.c >= S::TX)) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) put_tagged(x + f * plane + T.o + k * ld, act ? o[f] : 0.0, tag);
                }
            } else {
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const double z0 = MODE == 0 ? m[f] : a[f * S::PA];
                    if (EXACT && MODE == 0) kk[f] = cS * kk[f];
                    const double o = EXACT ? fma(cA, kk[f], cB * z0) : fma(cA, kk[f], z0);
                    if (!S::RESIDENT) dst[f * PT + q0 + k * RW] = act ? o : 0.0;
                    else if (act) dst[f * PT + q0 + k * RW] = o;
                    if (EXACT) D[k][f] = MODE == 0 ? kk[f] : D[k][f] + kk[f];
                    else D[k][f] = MODE == 0 ? cB * kk[f] : fma(cB, kk[f], D[k][f]);
                    if constexpr (EXACT && S::RESIDENT) {
                        if (MODE == 0 && f == 0) keep[q0 + k * RW] = o;
                    } else if constexpr (EXACT) {
                        if (f == 0 && r >= HALO && r < HALO + rows && T.c >= HALO && T.c < HALO + S::TX) {
                            // b.a4 and a3, then b.(a2 + a3), then b.a1
                            if (MODE == 0) keep[2 * S::TERM + term] = source_term(b, cS * m[0], gv), keep[S::TERM + term] = o;
                            else if (E == 2) keep[S::TERM + term] = source_term(b, o + keep[S::TERM + term], gv);
                            else keep[term] = source_term(b, o, gv);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) n[f] = m[f], m[f] = s[f], yv[f] = yn[f];
    }
}

// The 16-cell row segments of the tile (lattice of segment_sums in
// fk_kernels.cu) that hold a source cell, as row * (TX / 16) + segment: the
// others' terms are all zero and their partial sums stay at the zero the
// buffer was cleared to.
template <class S>
__device__ __forceinline__ void segment_list(uint16_t* list, int* count, const uint8_t* __restrict__ cells, int rows,
                                             int ld) {
    constexpr int SX = S::TX / 16;
    for (int i = threadIdx.x; i < rows * SX; i += blockDim.x) {
        const int r = i / SX, sx = i - r * SX;
        const uint8_t* c = cells + (long long)(r + HALO) * ld + HALO + sx * 16;
        bool any = false;
        for (int l = 0; l < 16; ++l) any = any || (c[l] & CELL_SOURCE);
        if (any) list[atomicAdd(count, 1)] = (uint16_t)i;
    }
}

// Partial sums of the listed segments, each by a half-warp in segment_sums'
// order; term(q) is the cell's term at window cell q, NaN counts as 0.  Every
// thread runs every round (the shuffles take whole warps).
template <class S, class Term>
__device__ __forceinline__ void segment_terms(const uint16_t* list, int count, double* __restrict__ row, int i0, int j0,
                                              int nsbx, Term term) {
    constexpr int SX = S::TX / 16;
    const int l = threadIdx.x & 15, h = threadIdx.x >> 4, nh = blockDim.x >> 4;
    for (int b0 = 0; b0 < count; b0 += nh) {
        if (b0 + (h & ~1) >= count) break;  // both halves of the warp are past the end
        const bool on = b0 + h < count;
        const int i = on ? list[b0 + h] : 0;
        const int r = i / SX, sx = i - r * SX;
        double s = 0.0;
        if (on) {
            const double t = term((r + HALO) * S::RW + HALO + sx * 16 + l);
            s = isnan(t) ? 0.0 : t;
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (on && l == 0) row[(long long)(i0 + r) * nsbx + (j0 / 16 + sx)] = s;
    }
}

// COPY: the job's parts in registers instead of read where they are needed.
// That ends the spills of 20 to 36 bytes of the instances with two and five
// rows a thread (exact mode 512 x 512 22.0 -> 20.9 us a step, 203 x 331 9.8 ->
// 9.1; reference mode 256 x 256 8.9 -> 8.6, 512 x 512 the same), but costs the exact
// instances that did not spill (384 x 384 15.7 -> 16.2) and, from shared
// memory, a batch (8.05 -> 8.24 ms).
template <class S, bool EXACT, bool COPY>
__device__ __forceinline__ void adj_run(const DevModel& P, const AdjJob& J) {
    constexpr int TX = S::TX, R = S::R, TYM = S::TYM;
    std::conditional_t<COPY, const DevGrid, const DevGrid&> g = J.g;
    std::conditional_t<COPY, const AdjRun, const AdjRun&> r = J.r;
    const double* __restrict__ gh = J.gh;
    const uint8_t* __restrict__ cells = J.cells;
    const uint8_t* __restrict__ adj = J.adj;
    const int ty = J.ty;
    constexpr int RW = S::RW;
    extern __shared__ double4 smem_raw[];
    __shared__ uint64_t bar;
    __shared__ int s_segs;
    __shared__ uint16_t segs[TYM * TX / 16];
    double* A = reinterpret_cast<double*>(smem_raw);
    double* B = A + 3 * S::PA - RW;
    double* C = A + 3 * (S::PA + S::PB) - 2 * RW;
    double* G = A + 3 * (S::PA + S::PB + S::PC) - RW;
    int2* ring = reinterpret_cast<int2*>(G + RW + S::PB);
    double* K3 = reinterpret_cast<double*>(ring + S::RING) - RW;  // a_3 on u (exact mode), rows 1 ..
    const int tile = blockIdx.x - J.tile0, by = tile / J.ntx, bx = tile - by * J.ntx;
    const int i0 = by * ty, j0 = bx * TX;
    const int rows = min(ty, g.nrows - i0);
    const long long off = (long long)i0 * g.ld + j0;
    const int nring = ring_table<S>(ring, g.ld, rows, i0, j0, g.nrows, J.ntx * TX);
    exp_table_init();
    if (threadIdx.x == 0) s_segs = 0;
    const uint32_t b = bulk_begin(&bar);
    __syncthreads();
    bulk_arrive(b, bulk_bytes<RW>(rows + 2 * HALO));
    __syncthreads();
    {
        const int nr = rows + 2 * HALO;
        for (int t = threadIdx.x; t < 3 * nr; t += blockDim.x) {
            const int f = t / nr, row = t - f * nr;
            bulk_row<RW>(b, A + f * S::PA + row * RW, r.zin + off + f * g.plane + (long long)row * g.ld);
        }
    }
    segment_list<S>(segs, &s_segs, cells + off, rows, g.ld);
    for (int q = threadIdx.x; q < 3 * S::PB; q += blockDim.x) B[RW + q] = 0.0;
    for (int q = threadIdx.x; q < 3 * S::PC; q += blockDim.x) C[2 * RW + q] = 0.0;
    Column T;
    {
        const int col = threadIdx.x / RW;
        T.c = threadIdx.x - col * RW;
        T.r0 = 1 + col * R;
        T.o = T.r0 * g.ld + T.c;
        T.bits = 0;
        if (T.r0 >= rows + 7) T.c = -1;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (T.c >= 1 && T.c < TX + 7 && T.r0 + k < rows + 7) {
                T.bits |= (unsigned)adj[off + T.o + k * g.ld] << (6 * k);
                G[(T.r0 + k) * RW + T.c] = gh[off + T.o + k * g.ld];
            }
        }
    }
    if (!bulk_wait_cta(b, r.fault)) return;
    __syncthreads();
    const int nsegs = s_segs;
    // the step's four states (k = 0 is the sweep's first, the latest in time)
    auto yptr = [&](int j) {  // y after j steps back
        return (j == 0 ? r.y_hi : (j == r.n ? r.y_lo : r.y_mid + (long long)(r.n - 1 - j) * r.stride)) + off;
    };
    auto point = [&](int k, int st) -> const double* {
        if (EXACT) return st == 3 ? yptr(k + 1) : r.pts + ((long long)k * r.pts_step + (2 - st)) * r.stride + off;
        return st == 0 ? yptr(k) : (st == 3 ? yptr(k + 1) : r.pts + (long long)k * r.pts_step * r.stride + off);
    };
    auto partial = [&](int group, int k) {
        return r.partial + ((long long)group * r.window + (r.row0 - k) % r.window) * r.nsb;
    };
    double D[R][3], yv[3];
    load_point<S>(T, 0, rows, g.ld, g.plane, point(0, 0), yv);
    for (int k = 0; k < r.n; ++k) {
        if (EXACT)
            segment_terms<S>(segs, nsegs, partial(2, k), i0, j0, r.nsbx,
                             [&](int q) { return ((P.dt_6) * A[q]) * G[q]; });
        adj_rows<3, S, 0, S::PA, S::PB, EXACT>(P, T, A, B, A, D, yv, point(k, 0), rows, g.ld, g.plane,
                                               EXACT ? P.dt : 0.5 * P.dt, EXACT ? P.dt_3 : 1.0 / 6.0 * P.dt,
                                               P.dt_6, K3, nullptr, nullptr, nullptr, 0);
        load_point<S>(T, 0, rows, g.ld, g.plane, point(k, 1), yv);
        __syncthreads();
        adj_rows<2, S, 1, S::PB, S::PC, EXACT>(P, T, B, C, A, D, yv, point(k, 1), rows, g.ld, g.plane, 0.5 * P.dt,
                                               EXACT ? P.dt_3 : 2.0 / 6.0 * P.dt, 0.0, nullptr, nullptr, nullptr,
                                               nullptr, 0);
        load_point<S>(T, 0, rows, g.ld, g.plane, point(k, 2), yv);
        __syncthreads();
        adj_rows<1, S, 1, S::PC, S::PB, EXACT>(P, T, C, B, A, D, yv, point(k, 2), rows, g.ld, g.plane,
                                               EXACT ? 0.5 * P.dt : P.dt, EXACT ? P.dt_6 : 2.0 / 6.0 * P.dt, 0.0,
                                               nullptr, nullptr, nullptr, nullptr, 0);
        load_point<S>(T, 0, rows, g.ld, g.plane, point(k, 3), yv);
        __syncthreads();
        if (EXACT) {
            segment_terms<S>(segs, nsegs, partial(0, k), i0, j0, r.nsbx, [&](int q) { return B[q] * G[q]; });
            segment_terms<S>(segs, nsegs, partial(1, k), i0, j0, r.nsbx, [&](int q) { return (C[q] + K3[q]) * G[q]; });
        }
        const bool end = k == r.n - 1;
        const unsigned long long tag = r.epoch + k + 1;
        Tagged* x = static_cast<Tagged*>(r.exchange) + (tag & 1) * (3 * g.plane) + off;
        adj_rows<0, S, 2, S::PB, S::PB, EXACT>(P, T, B, nullptr, A, D, yv, point(k, 3), rows, g.ld, g.plane, 0.0,
                                               1.0 / 6.0 * P.dt, 0.0, nullptr, nullptr, end ? r.zout + off : nullptr,
                                               end ? nullptr : x, tag);
        if (end) {
            __syncthreads();
        } else {
            load_point<S>(T, 0, rows, g.ld, g.plane, point(k + 1, 0), yv);
            if (!read_ring<S>(A, ring, nring, x, tag, g.plane, r.fault)) return;
        }
        // z_u . gh of the new z: the window's interior stays as it is until
        // the next step's last stage
        if (!EXACT)
            segment_terms<S>(segs, nsegs, partial(0, k), i0, j0, r.nsbx, [&](int q) { return A[q] * G[q]; });
    }
}

template <int TX, int R, int TYM, bool EXACT>
__global__ void __launch_bounds__(Shape<TX, R, TYM>::THREADS, 1) k_adj_run(const DevModel P, const AdjJob j) {
    adj_run<Shape<TX, R, TYM>, EXACT, !EXACT || R == 2 || R == 5>(P, j);
}

template <int TX, int R, int TYM, bool EXACT>
__global__ void __launch_bounds__(Shape<TX, R, TYM>::THREADS, 1)
    k_adj_jobs(const DevModel P, const RunJobs<AdjJob> jobs) {
    __shared__ AdjJob j;
    jobs.take(blockIdx.x, &j);
    adj_run<Shape<TX, R, TYM>, EXACT, false>(P, j);
}

// --------------------------------------------- per-step tiles, larger grids
//
// Where the tiles do not fit the device at once, a step is one launch of one
// CTA per SM, each taking tiles in turn; a tile's window arrives by bulk
// copies while the tile before it computes.  The stages are the sweeps'.  FP64
// issue and fixed latencies bound them (pipe 48 % busy forward, 41 % exact
// backward at 1536 x 1536, which also waits on DRAM for its points).  Forward,
// backward and exact backward us a step, with the preset kernels and here:
// 1024 x 768 52 and 43, 85 and 66; 2048 x 2048 218 and 199, 367 and 319, 405
// and 335.  (Prefetching the next tile's points into L2: 353 for the 335.)

// What a tile kernel's CTA goes through: tile i's place and window.
struct TileWalk {
    int ntx, tiles, ty;
    __device__ __forceinline__ int i0(int tile) const { return tile / ntx * ty; }
    __device__ __forceinline__ int j0(int tile) const { return tile % ntx * TileShapeBig::TX; }
};

// Issues the copies of the window of `tile` of state y into buffer A (its last
// readers are past a barrier), a few by every warp: by one warp, it fell 2 us a
// tile behind the others.  The copies may complete before thread 0 has posted
// their bytes: the barrier's phase ends with both.
__device__ __forceinline__ void fetch_tile(const DevGrid& g, const TileWalk& w, int tile, const double* y, double* A,
                                           uint32_t bar) {
    using S = TileShapeBig;
    const int i0 = w.i0(tile), nr = min(w.ty, g.nrows - i0) + 2 * HALO;
    const double* src = y + (long long)i0 * g.ld + w.j0(tile);
    bulk_arrive(bar, bulk_bytes<S::RW>(nr));
    const int t = (threadIdx.x & 31) * (S::THREADS / 32) + (threadIdx.x >> 5);
    static_assert(3 * (S::TYM + 2 * HALO) <= S::THREADS, "one copy per thread");
    if (t < 3 * nr) {
        const int f = t / nr, row = t - f * nr;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bulk_row<S::RW>(bar, A + f * S::PA + row * S::RW, src + f * g.plane + (long long)row * g.ld);
    }
}

// The barrier after a tile's first stage, with the outcome of its window's
// wait (one for the CTA): where the window did not arrive, as bulk_wait_cta,
// the fault word is set and the copies in flight (this tile's, and the next
// one's where it was fetched) waited for once more; the caller returns.
__device__ __forceinline__ bool window_arrived(bool ok, uint32_t bar, int n, bool next, unsigned* fault) {
    if (!__syncthreads_or(!ok)) return true;
    if (threadIdx.x == 0) atomicOr(fault, FAULT_TIMEOUT);
    bulk_drain<2>(bar, n, next ? n + 1 : n);
    return false;
}

// The flags of a thread's rows of a tile, loaded a tile ahead of their use
struct RowFlags {
    unsigned f[TileShapeBig::R];
    __device__ __forceinline__ void load(const DevGrid& g, const TileWalk& w, int tile, const Column& T, int c,
                                         const uint8_t* __restrict__ cells) {
        const int i0 = w.i0(tile), rows = min(w.ty, g.nrows - i0);
        const uint8_t* p = cells + (long long)i0 * g.ld + w.j0(tile) + T.o;
#pragma unroll
        for (int k = 0; k < TileShapeBig::R; ++k)
            f[k] = c >= 1 && c < TileShapeBig::TX + 7 && T.r0 + k < rows + 7 ? __ldg(p + k * g.ld) : 0u;
    }
    __device__ __forceinline__ unsigned bits() const {
        unsigned b = 0;
#pragma unroll
        for (int k = 0; k < TileShapeBig::R; ++k) b |= f[k] << (6 * k);
        return b;
    }
};

__device__ __forceinline__ Column tile_column(int ld) {
    Column T;
    const int col = threadIdx.x / TileShapeBig::RW;
    T.c = threadIdx.x - col * TileShapeBig::RW;
    T.r0 = 1 + col * TileShapeBig::R;
    T.o = T.r0 * ld + T.c;
    T.bits = 0;
    return T;
}

__global__ void __launch_bounds__(TileShapeBig::THREADS, 1)
    k_fwd_tile(const DevModel P, const DevGrid g, const double* __restrict__ gh, const uint8_t* __restrict__ cells,
               const FwdStep r, const TileWalk w) {
    using S = TileShapeBig;
    extern __shared__ double4 smem_raw[];
    __shared__ uint64_t bars[2];
    double* const W = reinterpret_cast<double*>(smem_raw);
    double* const B = W + 6 * S::PA - S::RW;
    double* const C = W + 3 * (2 * S::PA + S::PB) - 2 * S::RW;
    exp_table_init();
    const uint32_t bar = bulk_begin(&bars[0]);
    bulk_begin(&bars[1]);
    __syncthreads();
    Column T = tile_column(g.ld);
    const int c_all = T.c;
    double D[S::R][3];
    bool bad = false;
    int n = 0;
    RowFlags next;
    if ((int)blockIdx.x < w.tiles) {
        fetch_tile(g, w, blockIdx.x, r.src, W, bar);
        next.load(g, w, blockIdx.x, T, c_all, cells);
    }
    const double E0 = __ldg(r.E0), Eh = __ldg(r.Eh), E1 = __ldg(r.E1);
    for (int tile = blockIdx.x; tile < w.tiles; tile += gridDim.x, ++n) {
        const int i0 = w.i0(tile), rows = min(w.ty, g.nrows - i0);
        const long long off = (long long)i0 * g.ld + w.j0(tile);
        double* A = W + (n & 1) * 3 * S::PA;
        T.c = T.r0 < rows + 7 ? c_all : -1;
        T.bits = next.bits();
        const bool more = tile + (int)gridDim.x < w.tiles;
        if (more) {
            fetch_tile(g, w, tile + gridDim.x, r.src, W + (~n & 1) * 3 * S::PA, bar + 8 * (~n & 1));
            next.load(g, w, tile + gridDim.x, T, c_all, cells);
        }
        const bool ok = bulk_wait(bar + 8 * (n & 1), 1000000000ull, (unsigned)(n >> 1) & 1u);
        const double* ghs = gh + off;
        auto stage_out = [&](int st) { return r.stages ? r.stages + (long long)st * 3 * g.plane + off : nullptr; };
        fwd_rows<3, S, 0, S::PA, S::PB>(P, T, A, B, A, ghs, D, rows, g.ld, g.plane, E0, 0.5 * P.dt,
                                        1.0 / 6.0 * P.dt, stage_out(0), nullptr, 0, bad);
        if (!window_arrived(ok, bar, n, more, r.fault)) return;
        fwd_rows<2, S, 1, S::PB, S::PC>(P, T, B, C, A, ghs, D, rows, g.ld, g.plane, Eh, 0.5 * P.dt,
                                        1.0 / 3.0 * P.dt, stage_out(1), nullptr, 0, bad);
        __syncthreads();
        fwd_rows<1, S, 1, S::PC, S::PB>(P, T, C, B, A, ghs, D, rows, g.ld, g.plane, Eh, P.dt,
                                        1.0 / 3.0 * P.dt, stage_out(2), nullptr, 0, bad);
        __syncthreads();
        if (r.dst)
            fwd_rows<0, S, 2, S::PB, S::PB>(P, T, B, nullptr, A, ghs, D, rows, g.ld, g.plane, E1, 0.0,
                                            P.dt_6, r.dst + off, nullptr, 0, bad);
        __syncthreads();  // B and A are free
    }
    if (bad) atomicOr(r.fault, FAULT_NAN);
}

template <bool EXACT>
__global__ void __launch_bounds__(TileShapeBig::THREADS, 1)
    k_adj_tile(const DevModel P, const DevGrid g, const double* __restrict__ gh, const uint8_t* __restrict__ adj,
               const uint8_t* __restrict__ segs, const AdjStep r, const TileWalk w) {
    using S = TileShapeBig;
    extern __shared__ double4 smem_raw[];
    __shared__ uint64_t bars[2];
    double* const W = reinterpret_cast<double*>(smem_raw);
    double* const B = W + 6 * S::PA - S::RW;
    double* const C = W + 3 * (2 * S::PA + S::PB) - 2 * S::RW;
    double* const terms = W + 3 * (2 * S::PA + S::PB + S::PC);
    exp_table_init();
    const uint32_t bar = bulk_begin(&bars[0]);
    bulk_begin(&bars[1]);
    __syncthreads();
    Column T = tile_column(g.ld);
    const int c_all = T.c;
    double D[S::R][3], yv[3];
    int n = 0;
    RowFlags next;
    if ((int)blockIdx.x < w.tiles) {
        fetch_tile(g, w, blockIdx.x, r.zin, W, bar);
        next.load(g, w, blockIdx.x, T, c_all, adj);
    }
    for (int tile = blockIdx.x; tile < w.tiles; tile += gridDim.x, ++n) {
        const int i0 = w.i0(tile), j0 = w.j0(tile), rows = min(w.ty, g.nrows - i0);
        const long long off = (long long)i0 * g.ld + j0;
        double* A = W + (n & 1) * 3 * S::PA;
        T.c = T.r0 < rows + 7 ? c_all : -1;
        T.bits = next.bits();
        load_point<S>(T, 0, rows, g.ld, g.plane, r.y[0] + off, yv);
        const bool more = tile + (int)gridDim.x < w.tiles;
        if (more) {
            fetch_tile(g, w, tile + gridDim.x, r.zin, W + (~n & 1) * 3 * S::PA, bar + 8 * (~n & 1));
            next.load(g, w, tile + gridDim.x, T, c_all, adj);
        }
        const bool ok = bulk_wait(bar + 8 * (n & 1), 1000000000ull, (unsigned)(n >> 1) & 1u);
        const double* ghs = gh + off;
        adj_rows<3, S, 0, S::PA, S::PB, EXACT>(P, T, A, B, A, D, yv, r.y[0] + off, rows, g.ld, g.plane,
                                               EXACT ? P.dt : 0.5 * P.dt, EXACT ? P.dt_3 : 1.0 / 6.0 * P.dt,
                                               P.dt_6, terms, ghs, nullptr, nullptr, 0);
        load_point<S>(T, 0, rows, g.ld, g.plane, r.y[1] + off, yv);
        if (!window_arrived(ok, bar, n, more, r.fault)) return;
        adj_rows<2, S, 1, S::PB, S::PC, EXACT>(P, T, B, C, A, D, yv, r.y[1] + off, rows, g.ld, g.plane, 0.5 * P.dt,
                                               EXACT ? P.dt_3 : 2.0 / 6.0 * P.dt, 0.0, terms, ghs, nullptr,
                                               nullptr, 0);
        load_point<S>(T, 0, rows, g.ld, g.plane, r.y[2] + off, yv);
        __syncthreads();
        adj_rows<1, S, 1, S::PC, S::PB, EXACT>(P, T, C, B, A, D, yv, r.y[2] + off, rows, g.ld, g.plane,
                                               EXACT ? 0.5 * P.dt : P.dt, EXACT ? P.dt_6 : 2.0 / 6.0 * P.dt, 0.0,
                                               terms, ghs, nullptr, nullptr, 0);
        load_point<S>(T, 0, rows, g.ld, g.plane, r.y[3] + off, yv);
        __syncthreads();
        adj_rows<0, S, 2, S::PB, S::PB, EXACT>(P, T, B, nullptr, A, D, yv, r.y[3] + off, rows, g.ld, g.plane, 0.0,
                                               1.0 / 6.0 * P.dt, 0.0, terms, ghs, r.zout + off, nullptr, 0);
        __syncthreads();
        // partial sums of the row segments with a source, as segment_terms
        constexpr int SX = S::TX / 16;
        const int l = threadIdx.x & 15, h = threadIdx.x >> 4, nh = blockDim.x >> 4;
        for (int s0 = 0; s0 < rows * SX; s0 += nh) {
            const int i = s0 + h, row = i / SX, sx = i - row * SX;
            const long long at = (long long)(i0 + row) * r.nsbx + (j0 / 16 + sx);
            const bool on = i < rows * SX && __ldg(segs + at);
            if (!__any_sync(0xffffffffu, on)) continue;
            for (int gr = 0; gr < (EXACT ? 3 : 1); ++gr) {
                double s = on ? terms[gr * S::TERM + row * S::TX + sx * 16 + l] : 0.0;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (on && l == 0) r.row[gr][at] = s;
            }
        }
        if (EXACT) __syncthreads();  // the next tile's first stage writes terms
    }
}

// ------------------------------------------------------- midpoint states
//
// The midpoint states of r.n backward steps (cu-G:1244-1301) in one launch:
// they depend on the stored states only, so the steps of a sweep's chunk are
// all made before it.  A CTA takes one tile of one run of steps, walking back
// in time: the state and f of a step's later end are the earlier end of the
// step before it, so each step costs two evaluations and one window load,
// issued a step ahead.  Per-step launches took 14 us a step at 512 x 512,
// waiting for their operands; this takes 6.6 (2048 x 2048: 207 and 133), the
// FP64 pipe 50 % and the issue slots 64 % busy.
//   y(1/3) = cubic Hermite of (ya, fa, yb, fb) at 1/3,
//   yh     = partial quartic at 1/2 + (27/64) dt f(y(1/3), E(t + dt/3)).
// One barrier a step: the y(1/3) buffers alternate, every warp issues a few of
// the window's copies, and every thread waits for them itself (with barriers at
// each of these points, 30 % of the warps' time went into them).
struct MidShape {
    static constexpr int TX = 64, R = 2, TY = 16, H = 2, RW = TX + 2 * HALO;
    static constexpr int LW = TX + 2;                 // columns evaluated: the tile and one cell around it
    static constexpr int PW = (TY + 2 * H) * RW;      // a window: rows -2 .. TY + 1
    static constexpr int THREADS = (LW * ((TY + 2) / R) + 31) / 32 * 32;
    static constexpr size_t SMEM = sizeof(double) * (size_t)(3 * 3 * PW + 2 * 3 * PW + PW);
    static_assert((TY + 2) % R == 0 && THREADS <= 640, "96 registers per thread");
    static_assert(3 * (TY + 2 * H) <= THREADS, "one window copy per thread");
};

// f at the thread's cell of row k (window row r) of buffer Y from its column
// values; as in fwd_rows
__device__ __forceinline__ void mid_field(const DevModel& P, unsigned b, const double* Y, const double* g,
                                          double E, double (&kk)[3]) {
    constexpr int RW = MidShape::RW, PW = MidShape::PW;
    const double* pn = Y + ((b & CELL_N) ? RW : -RW);
    const double* ps = Y + ((b & CELL_S) ? -RW : RW);
    const double* pw = Y + ((b & CELL_W) ? 1 : -1);
    const double* pe = Y + ((b & CELL_E) ? -1 : 1);
    double y[3], t[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) y[f] = Y[f * PW];
#pragma unroll
    for (int f = 0; f < 3; ++f) t[f] = lap4(pn[f * PW], ps[f * PW], pw[f * PW], pe[f * PW], y[f]);
    double gv = 0.0;
    if (b & CELL_SOURCE) gv = *g;
    fk_field(P, y, t, E, gv, kk[0], kk[1], kk[2]);
}

__device__ __forceinline__ void mid_run(const DevModel& P, const HermiteW& hw, const MidJob& J) {
    using S = MidShape;
    const DevGrid& g = J.g;
    const MidRun& r = J.r;
    const double* __restrict__ gh = J.gh;
    const uint8_t* __restrict__ cells = J.cells;
    constexpr int RW = S::RW, PW = S::PW, R = S::R;
    extern __shared__ double4 smem_raw[];
    __shared__ uint64_t bars[3];
    double* W = reinterpret_cast<double*>(smem_raw);  // three windows in turn
    double* Y3 = W + 9 * PW;                          // two buffers in turn
    double* G = Y3 + 6 * PW;
    const int bx = (blockIdx.x - J.tile0) % J.ntx, t0 = (blockIdx.x - J.tile0) / J.ntx;
    const int i0 = t0 % J.nty * S::TY, j0 = bx * S::TX;
    const int rows = min(S::TY, g.nrows - i0);
    // window origin: logical (i0 - 2, j0 - 4) = padded (i0 + 2, j0)
    const long long off = (long long)(i0 + HALO - S::H) * g.ld + j0;
    const int k0 = t0 / J.nty * J.per, k1 = min(k0 + J.per, r.n);  // steps k0 .. k1 - 1
    if (k0 >= k1) return;
    exp_table_init();
    const uint32_t bar = bulk_begin(&bars[0]);
    bulk_begin(&bars[1]);
    bulk_begin(&bars[2]);
    __syncthreads();
    const int nr = rows + 2 * S::H;
    // the window of y after j steps back into buffer (j - k0) % 3 (as
    // fetch_tile); its barrier's parity is (j - k0) / 3 mod 2
    auto fetch = [&](int j) {
        const int u = (j - k0) % 3;
        const double* src =
            (j == 0 ? r.y_hi : (j == r.n ? r.y_lo : r.y_mid + (long long)(r.n - 1 - j) * r.stride)) + off;
        bulk_arrive(bar + 8 * u, bulk_bytes<RW>(nr));
        const int t = (threadIdx.x & 31) * (S::THREADS / 32) + (threadIdx.x >> 5);
        if (t < 3 * nr) {
            const int f = t / nr, row = t - f * nr;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bulk_row<RW>(bar + 8 * u, W + (3 * u + f) * PW + row * RW, src + f * g.plane + (long long)row * g.ld);
        }
    };
    fetch(k0);
    fetch(k0 + 1);
    const int col = threadIdx.x / S::LW;
    const int c = HALO - 1 + threadIdx.x - col * S::LW, r0 = 1 + col * R;
    unsigned bits = 0;
    double fb[R][3];
#pragma unroll
    for (int k = 0; k < R; ++k)
        if (r0 + k < rows + 3) {
            bits |= (unsigned)cells[off + (long long)(r0 + k) * g.ld + c] << (6 * k);
            G[(r0 + k) * RW + c] = gh[off + (long long)(r0 + k) * g.ld + c];
        }
    if (!bulk_wait_cta(bar, r.fault)) {
        bulk_drain<3>(bar, 1, 1);  // the second window is in flight too
        return;
    }
#pragma unroll
    for (int k = 0; k < R; ++k)
        if (r0 + k < rows + 3) {
            const int q = (r0 + k) * RW + c;
            mid_field(P, bits >> (6 * k), W + q, G + q, __ldg(r.Et - k0), fb[k]);
        }
    for (int k = k0; k < k1; ++k) {
        const int ub = (k - k0) % 3, ua = (k + 1 - k0) % 3;
        // the window after next into the buffer that the step before last read
        // (its readers are past the last step's barrier)
        if (k + 2 <= k1) fetch(k + 2);
        const double Ea = __ldg(r.Et - k - 1), E3 = __ldg(r.E3 - k);
        const bool ok = bulk_wait(bar + 8 * ua, 1000000000ull, (unsigned)((k + 1 - k0) / 3) & 1u);
        const double* YA = W + 3 * ua * PW;
        const double* YB = W + 3 * ub * PW;
        double* T3 = Y3 + 3 * ((k - k0) & 1) * PW;
        double qv[R][3];
#pragma unroll
        for (int u = 0; u < R; ++u)
            if (r0 + u < rows + 3) {
                const int q = (r0 + u) * RW + c;
                double fa[3];
                mid_field(P, bits >> (6 * u), YA + q, G + q, Ea, fa);
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const double m0 = fa[f] * P.dt, m1 = fb[u][f] * P.dt;
                    const double x0 = YA[f * PW + q], x1 = YB[f * PW + q];
                    T3[f * PW + q] = hermite4(hw.c3, x0, m0, x1, m1);
                    qv[u][f] = hermite4(hw.c4, x0, m0, x1, m1);
                    fb[u][f] = fa[f];
                }
            }
        if (__syncthreads_or(!ok)) {
            // a window did not arrive in time: as bulk_wait_cta, once more for
            // the copies in flight, then out
            if (threadIdx.x == 0) atomicOr(r.fault, FAULT_TIMEOUT);
            bulk_drain<3>(bar, k + 1 - k0, min(k + 2, k1) - k0);
            return;
        }
        double* yh = r.yh + (long long)k * r.stride + off;
#pragma unroll
        for (int u = 0; u < R; ++u)
            if (c >= HALO && c < HALO + S::TX && r0 + u >= S::H && r0 + u < S::H + rows) {
                const int q = (r0 + u) * RW + c;
                double m2[3];
                mid_field(P, bits >> (6 * u), T3 + q, G + q, E3, m2);
#pragma unroll
                for (int f = 0; f < 3; ++f)
                    yh[f * g.plane + (long long)(r0 + u) * g.ld + c] = fma(hw.c2, m2[f] * P.dt, qv[u][f]);
            }
    }
}

__global__ void __launch_bounds__(MidShape::THREADS, 1) k_mid_run(const DevModel P, const HermiteW hw, const MidJob j) {
    mid_run(P, hw, j);
}

__global__ void __launch_bounds__(MidShape::THREADS, 1)
    k_mid_jobs(const DevModel P, const HermiteW hw, const RunJobs<MidJob> jobs) {
    __shared__ MidJob j;
    jobs.take(blockIdx.x, &j);
    mid_run(P, hw, j);
}

}  // namespace

#define X(id, a, b, c) \
    case id: { using S = Shape<a, b, c>; DO(S); } break;

constexpr int kRunShapes = 8;
struct ShapeInfo {
    int tx, R, tym, rw, threads;
    // a step's cost on tiles of `rows` rows: per stage, the evaluations (a
    // warp's row, by FP64 issue) or the depth of a thread's column, whichever
    // is longer, and something for the depth in any case
    double cost(int rows) const {
        double c = 0;
        for (int e = 3; e >= 0; --e) c += std::max((double)rw * (rows + 2 * e) / 32.0 * 62.0, R * 420.0) + R * 40.0;
        return c;
    }
    int threads_for(int rows) const { return std::min(threads, (rw * ((rows + 6 + R - 1) / R) + 31) / 32 * 32); }
};
static ShapeInfo shape_info(int id) {
    switch (id) {
#define DO(S) return {S::TX, S::R, S::TYM, S::RW, S::THREADS}
        FKADJ_RUN_LIST(X)
#undef DO
    }
    return {};
}

RunShape run_shape(const DevGrid& g, int sms) {
    RunShape best;
    double best_cost = 0;
    for (int id = 0; id < kRunShapes; ++id) {
        const ShapeInfo f = shape_info(id);
        const int ntx = (g.ncols + f.tx - 1) / f.tx;
        if (ntx > sms) continue;
        // at least 4 rows: a tile's halo is its direct neighbours' cells
        const int rows = std::max(HALO, (g.nrows + sms / ntx - 1) / (sms / ntx));
        if (rows > f.tym) continue;
        const double cost = f.cost(rows);
        if (best.id < 0 || cost < best_cost) {
            best_cost = cost;
            best = {id, f.tx, rows, ntx, (g.nrows + rows - 1) / rows, f.threads_for(rows)};
        }
    }
    return best;
}

// Launches of several problems: each cooperative launch occupies the device for
// as long as its longest sweep, and two do not overlap, so small grids one
// after the other leave most SMs idle.  Ten uneven gradients to 256 x 256 x
// 150: 16.1 ms a step at a time with the tick kernels, 8.1 packed.
//
// How n problems' tiles share launches of at most `sms` tiles and kRunJobs
// problems: their shape, each one's launch, and the rows of a tile in each.
struct RunPacking {
    int id = -1, bins = 0;
    std::vector<int> bin, rows;
    double cost = 0;
};

// The packing of shape `id`, or bins = 0 where a grid does not fit in it: the
// largest problem to the emptiest of as few launches as hold them all, then
// in each launch as few rows a tile as still fit.
template <class Job>
static RunPacking pack_shape(const Job* j, int n, int id, int sms) {
    const ShapeInfo f = shape_info(id);
    auto tiles = [&](int q, int rows) {
        return ((j[q].g.ncols + f.tx - 1) / f.tx) * ((j[q].g.nrows + rows - 1) / rows);
    };
    RunPacking p;
    std::vector<int> order(n);
    long long total = 0;
    for (int q = 0; q < n; ++q) {
        order[q] = q;
        total += tiles(q, f.tym);
        if (tiles(q, f.tym) > sms) return p;
    }
    std::sort(order.begin(), order.end(), [&](int a, int b) { return tiles(a, f.tym) > tiles(b, f.tym); });
    std::vector<int> load, count;
    for (int bins = std::max((int)((total + sms - 1) / sms), (n + kRunJobs - 1) / kRunJobs);; ++bins) {
        load.assign(bins, 0);
        count.assign(bins, 0);
        p.bin.assign(n, 0);
        bool fits = true;
        for (int q : order) {
            int b = -1;
            for (int c = 0; c < bins; ++c)
                if (count[c] < kRunJobs && (b < 0 || load[c] < load[b])) b = c;
            load[b] += tiles(q, f.tym);
            ++count[b];
            p.bin[q] = b;
            fits = fits && load[b] <= sms;
        }
        if (!fits) continue;  // ends at one problem per launch at the latest
        p.bins = bins;
        break;
    }
    p.id = id;
    for (int b = 0; b < p.bins; ++b) {
        int rows = f.tym;
        for (; rows > HALO; --rows) {
            int t = 0;
            for (int q = 0; q < n; ++q)
                if (p.bin[q] == b) t += tiles(q, rows - 1);
            if (t > sms) break;
        }
        p.rows.push_back(rows);
        p.cost += f.cost(rows);
    }
    return p;
}

// Runs n jobs packed: launch(id, jobs of one launch, threads, tiles).  Where
// no shape takes all the grids, in two parts (run_shape has one for each).
template <class Job, class Launch>
static cudaError_t run_packed(const Job* j, int n, int sms, Launch&& launch) {
    if (n <= 0) return cudaSuccess;
    RunPacking best;
    for (int id = 0; id < kRunShapes; ++id) {
        RunPacking p = pack_shape(j, n, id, sms);
        if (p.bins > 0 && (best.bins == 0 || p.cost < best.cost)) best = std::move(p);
    }
    if (best.bins == 0) {
        if (n == 1) return cudaErrorInvalidValue;
        const cudaError_t e = run_packed(j, n / 2, sms, launch);
        return e ? e : run_packed(j + n / 2, n - n / 2, sms, launch);
    }
    const ShapeInfo f = shape_info(best.id);
    for (int b = 0; b < best.bins; ++b) {
        RunJobs<Job> jobs;
        jobs.n = 0;
        int tiles = 0;
        for (int q = 0; q < n; ++q) {
            if (best.bin[q] != b) continue;
            Job& k = jobs.job[jobs.n++];
            k = j[q];
            const int nty = (k.g.nrows + best.rows[b] - 1) / best.rows[b];
            k.ty = std::max(HALO, (k.g.nrows + nty - 1) / nty);
            k.ntx = (k.g.ncols + f.tx - 1) / f.tx;
            k.tile0 = tiles;
            tiles += k.ntx * ((k.g.nrows + k.ty - 1) / k.ty);
        }
        if (const cudaError_t e = launch(best.id, jobs, f.threads_for(best.rows[b]), tiles)) return e;
    }
    return cudaSuccess;
}

size_t run_exchange_bytes(const DevGrid& g) { return 2 * 3 * (size_t)g.plane * sizeof(Tagged); }

cudaError_t run_init() {
    cudaError_t e = cudaFuncSetAttribute(k_mid_run, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MidShape::SMEM);
    if (!e) e = cudaFuncSetAttribute(k_mid_jobs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MidShape::SMEM);
    const int big = (int)TileShapeBig::SMEM;
    if (!e) e = cudaFuncSetAttribute(k_fwd_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
    if (!e) e = cudaFuncSetAttribute(k_adj_tile<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
    if (!e) e = cudaFuncSetAttribute(k_adj_tile<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
#undef X
#define N_(K, smem) \
    if (!e) e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem))
#define X(id, a, b, c)                                                    \
    N_((k_fwd_run<a, b, c>), (Shape<a, b, c>::SMEM));                  \
    N_((k_fwd_jobs<a, b, c>), (Shape<a, b, c>::SMEM));           \
    N_((k_adj_run<a, b, c, false>), (Shape<a, b, c>::SMEM));           \
    N_((k_adj_jobs<a, b, c, false>), (Shape<a, b, c>::SMEM));    \
    N_((k_adj_run<a, b, c, true>), (Shape<a, b, c>::SMEM_EXACT));      \
    N_((k_adj_jobs<a, b, c, true>), (Shape<a, b, c>::SMEM_EXACT));
    FKADJ_RUN_LIST(X)
#undef X
#undef N_
    return e;
}

template <class K, class Jobs>
static cudaError_t launch_run(K kernel, int tiles, int threads, size_t smem, cudaStream_t st, const DevModel& P,
                              const Jobs& jobs) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P, jobs);
}

template <class Job>
static Job placed(const RunShape& s, Job j) {
    j.ty = s.rows;
    j.ntx = s.ntx;
    j.tile0 = 0;
    return j;
}

cudaError_t launch_fwd_run(const RunShape& s, const DevModel& P, const FwdJob& j, cudaStream_t st) {
    if (j.r.n <= 0) return cudaSuccess;
    switch (s.id) {
#define X(id, a, b, c) \
    case id: return launch_run(k_fwd_run<a, b, c>, s.tiles(), s.threads, Shape<a, b, c>::SMEM, st, P, placed(s, j));
        FKADJ_RUN_LIST(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_adj_run(const RunShape& s, bool exact, const DevModel& P, const AdjJob& j, cudaStream_t st) {
    if (j.r.n <= 0) return cudaSuccess;
    const AdjJob q = placed(s, j);
    switch (s.id) {
#define X(id, a, b, c)                                                                                                 \
    case id:                                                                                                           \
        return exact ? launch_run(k_adj_run<a, b, c, true>, s.tiles(), s.threads, Shape<a, b, c>::SMEM_EXACT, st, P, q) \
                     : launch_run(k_adj_run<a, b, c, false>, s.tiles(), s.threads, Shape<a, b, c>::SMEM, st, P, q);
        FKADJ_RUN_LIST(X)
#undef X
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_fwd_jobs(const DevModel& P, const FwdJob* j, int n, int sms, cudaStream_t st, int64_t* launches) {
    return run_packed(j, n, sms, [&](int id, const RunJobs<FwdJob>& jobs, int threads, int tiles) {
        ++*launches;
        switch (id) {
#define X(id, a, b, c) \
    case id: return launch_run(k_fwd_jobs<a, b, c>, tiles, threads, Shape<a, b, c>::SMEM, st, P, jobs);
            FKADJ_RUN_LIST(X)
#undef X
        }
        return cudaErrorInvalidValue;
    });
}

cudaError_t launch_adj_jobs(bool exact, const DevModel& P, const AdjJob* j, int n, int sms, cudaStream_t st,
                            int64_t* launches) {
    return run_packed(j, n, sms, [&](int id, const RunJobs<AdjJob>& jobs, int threads, int tiles) {
        ++*launches;
        switch (id) {
#define X(id, a, b, c)                                                                                           \
    case id:                                                                                                     \
        return exact ? launch_run(k_adj_jobs<a, b, c, true>, tiles, threads, Shape<a, b, c>::SMEM_EXACT, st, P, jobs) \
                     : launch_run(k_adj_jobs<a, b, c, false>, tiles, threads, Shape<a, b, c>::SMEM, st, P, jobs);
            FKADJ_RUN_LIST(X)
#undef X
        }
        return cudaErrorInvalidValue;
    });
}

// Rows per tile of the per-step tile kernels: the fewest waves of CTAs, then
// the least work per wave (a tile's cost goes with its rows and the halo's).
static TileWalk tile_walk(const DevGrid& g, int sms) {
    using S = TileShapeBig;
    TileWalk w{(g.ncols + S::TX - 1) / S::TX, 0, 0};
    long long best = -1;
    for (int ty = HALO; ty <= S::TYM; ++ty) {
        const int tiles = w.ntx * ((g.nrows + ty - 1) / ty);
        const long long cost = (long long)((tiles + sms - 1) / sms) * (4 * ty + 12 + 16);
        if (best < 0 || cost <= best) best = cost, w.ty = ty, w.tiles = tiles;
    }
    return w;
}

void run_tile(const DevGrid& g, const RunShape& s, int sms, bool midpoint, int tile[3]) {
    const int mid[3] = {MidShape::TX, MidShape::TY, MidShape::THREADS};
    const int run[3] = {s.tx, s.rows, s.threads};
    const int big[3] = {TileShapeBig::TX, tile_walk(g, sms).ty, TileShapeBig::THREADS};
    const int* t = midpoint ? mid : (s.id >= 0 ? run : big);
    std::copy(t, t + 3, tile);
}

cudaError_t launch_fwd_tile(const DevModel& P, const DevGrid& g, const double* gh, const uint8_t* cells,
                            const FwdStep& r, int sms, cudaStream_t st) {
    using S = TileShapeBig;
    const TileWalk w = tile_walk(g, sms);
    k_fwd_tile<<<std::min(sms, w.tiles), S::THREADS, S::SMEM, st>>>(P, g, gh, cells, r, w);
    return cudaGetLastError();
}

cudaError_t launch_adj_tile(bool exact, const DevModel& P, const DevGrid& g, const double* gh, const uint8_t* adj,
                            const uint8_t* segs, const AdjStep& r, int sms, cudaStream_t st) {
    using S = TileShapeBig;
    const TileWalk w = tile_walk(g, sms);
    if (exact) k_adj_tile<true><<<std::min(sms, w.tiles), S::THREADS, S::SMEM, st>>>(P, g, gh, adj, segs, r, w);
    else k_adj_tile<false><<<std::min(sms, w.tiles), S::THREADS, S::SMEM, st>>>(P, g, gh, adj, segs, r, w);
    return cudaGetLastError();
}

// Fills in where n midpoint jobs' tiles lie, one after the other; returns
// their CTAs.  Runs of steps per CTA: the fewest evaluations (per steps cost 2
// per + 1) over whole waves of CTAs, one per SM.
static int place_mid(MidJob* j, int n, int sms) {
    using S = MidShape;
    int most = 1, per = 1;
    for (int q = 0; q < n; ++q) {
        j[q].ntx = (j[q].g.ncols + S::TX - 1) / S::TX;
        j[q].nty = (j[q].g.nrows + S::TY - 1) / S::TY;
        most = std::max(most, j[q].r.n);
    }
    auto ctas = [&](int q, int p) { return j[q].ntx * j[q].nty * ((j[q].r.n + p - 1) / p); };
    long long best = -1;
    for (int p = 1; p <= most; ++p) {
        long long c = 0;
        for (int q = 0; q < n; ++q) c += ctas(q, p);
        const long long cost = (c + sms - 1) / sms * (2 * p + 1);
        if (best < 0 || cost <= best) best = cost, per = p;
    }
    int tile0 = 0;
    for (int q = 0; q < n; ++q) {
        j[q].per = per;
        j[q].tile0 = tile0;
        tile0 += ctas(q, per);
    }
    return tile0;
}

cudaError_t launch_mid_run(const DevModel& P, const HermiteW& hw, const MidJob& j, int sms, cudaStream_t st) {
    if (j.r.n <= 0) return cudaSuccess;
    MidJob q = j;
    const int ctas = place_mid(&q, 1, sms);
    k_mid_run<<<ctas, MidShape::THREADS, MidShape::SMEM, st>>>(P, hw, q);
    return cudaGetLastError();
}

cudaError_t launch_mid_jobs(const DevModel& P, const HermiteW& hw, const MidJob* j, int n, int sms, cudaStream_t st,
                            int64_t* launches) {
    for (int q0 = 0; q0 < n; q0 += kRunJobs) {
        RunJobs<MidJob> jobs;
        jobs.n = std::min(kRunJobs, n - q0);
        std::copy(j + q0, j + q0 + jobs.n, jobs.job);
        const int ctas = place_mid(jobs.job, jobs.n, sms);
        ++*launches;
        k_mid_jobs<<<ctas, MidShape::THREADS, MidShape::SMEM, st>>>(P, hw, jobs);
        if (const cudaError_t e = cudaGetLastError()) return e;
    }
    return cudaSuccess;
}

}  // namespace fkadj
