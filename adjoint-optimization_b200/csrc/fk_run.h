// fk_run.h -- sweeps of many time steps in one launch, for grids whose tiles
// fit the device at once (fk_run.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "fk_kernels.h"

namespace fkadj {

// Per-cell flags of the sweep kernels (a byte per padded cell, 0 at holes and
// off the grid): which neighbours are missing and mirrored, as the reference's
// stencil does (S: south missing and north present, E likewise; a cell that
// lacks two opposite neighbours turns into a hole, which no fixed flags
// describe: grids with such cells are not swept), and where the source is.
constexpr unsigned CELL_N = 1, CELL_S = 2, CELL_W = 4, CELL_E = 8, CELL_ACTIVE = 16, CELL_SOURCE = 32;

// The adjoint sweeps' flags (a byte per padded cell): the neighbours that
// mirror this cell, which the transposed stencil counts twice.
constexpr unsigned CELL_2N = 1, CELL_2S = 2, CELL_2W = 4, CELL_2E = 8, CELL_ACTIVE_ADJ = 16;

// How a grid is cut for a sweep: tiles of tx columns by `rows` rows, one CTA
// of `threads` threads each, R rows of a column per thread.
struct RunShape {
    int id = -1;  // kernel instance (-1: the grid does not fit, per-step launches)
    int tx = 0, rows = 0, ntx = 0, nty = 0, threads = 0;
    int tiles() const { return ntx * nty; }
};

// Tiles of a swept grid's launches: columns, rows, threads of a sweep (s.id >=
// 0) or of the tile kernels, or of the midpoint kernel.
void run_tile(const DevGrid& g, const RunShape& s, int sms, bool midpoint, int tile[3]);

// The shape for grid g on a device with `sms` multiprocessors (id -1: none).
RunShape run_shape(const DevGrid& g, int sms);
cudaError_t run_init();

// Bytes of the exchange area of grid g's sweeps (zeroed once; see k_fwd_run).
size_t run_exchange_bytes(const DevGrid& g);

// One forward sweep of n steps from state src.  The state after step k
// (0-based) goes to `last` for k = n - 1; of the others, when out is non-null,
// those after `first` steps and every `every` more go to out, out + stride,
// and so on.  None of them is src.
struct FwdRun {
    const double* src;
    double* last;
    double* out;
    double* stages;         // stage states Y2, Y3, Y4 of step k to stages + (3 k + 0 .. 2) * stride (null: not kept)
    long long stride;
    int n, first, every;
    const double *Et, *Eh;  // samples: step k takes Et[k], Eh[k], Et[k + 1]
    void* exchange;
    unsigned long long epoch;  // steps of all the sweeps before this one: the exchange's tags are never reset
    unsigned* fault;
};
constexpr unsigned FAULT_TIMEOUT = 1, FAULT_NAN = 2;

// One backward sweep of n steps from zin (z, resp. lambda, at the later end) to
// zout, two distinct states.  Step k takes the state from the later end back:
// y_hi for k = 0, y_mid + (n - 1 - k) * stride, and y_lo after the last step.
// pts: the points between them, step k's at pts + k * pts_step * stride (reference mode:
// the midpoint state) or, in the exact mode, its stage states Y2, Y3, Y4 at
// the three states from pts + k * pts_step * stride.
// Partial z.gh sums on the row-segment lattice (nsb = nsbx x grid rows per
// row of results): step k's go to row (row0 - k) mod window of group 0 of
// `partial`; exact mode: b.a1, b.(a2 + a3), b.a4 to groups 0, 1, 2 (window
// rows each).  Segments without a source cell are not written.
struct AdjRun {
    const double* zin;
    double* zout;
    const double *y_hi, *y_mid, *y_lo, *pts;
    long long stride;
    int pts_step, n;
    double* partial;
    long long nsb;
    int nsbx, row0, window;
    void* exchange;
    unsigned long long epoch;
    unsigned* fault;
};
// Midpoint states of n backward steps (reference mode), step k's to yh + k *
// stride; y_hi, y_mid, y_lo as in AdjRun.  Et, E3: the samples at the later end
// of step 0 and of step 0's third; step k takes Et[-k], Et[-k - 1], E3[-k].
struct MidRun {
    const double *y_hi, *y_mid, *y_lo;
    double* yh;
    long long stride;
    int n;
    const double *Et, *E3;
    unsigned* fault;
};
// The sweeps of one launch: a problem's grid and tables, its sweep, and where
// its tiles lie (filled in by the launch functions).  Sweeps of several
// problems of one model share a launch where their tiles fit the device
// together; none waits for another's.
struct FwdJob {
    DevGrid g;
    const double* gh;
    const uint8_t* cells;
    FwdRun r;
    int ty, ntx, tile0;
};
struct AdjJob {
    DevGrid g;
    const double* gh;
    const uint8_t *cells, *adj;
    AdjRun r;
    int ty, ntx, tile0;
};
struct MidJob {
    DevGrid g;
    const double* gh;
    const uint8_t* cells;
    MidRun r;
    int per, ntx, nty, tile0;
};

// One problem's sweep, cut as s.
cudaError_t launch_fwd_run(const RunShape& s, const DevModel& P, const FwdJob& j, cudaStream_t st);
cudaError_t launch_adj_run(const RunShape& s, bool exact, const DevModel& P, const AdjJob& j, cudaStream_t st);
cudaError_t launch_mid_run(const DevModel& P, const HermiteW& hw, const MidJob& j, int sms, cudaStream_t st);

// n problems' sweeps (each grid fits the device: run_shape), in as few
// launches as their tiles need; adds those to *launches.
cudaError_t launch_fwd_jobs(const DevModel& P, const FwdJob* j, int n, int sms, cudaStream_t st, int64_t* launches);
cudaError_t launch_adj_jobs(bool exact, const DevModel& P, const AdjJob* j, int n, int sms, cudaStream_t st,
                            int64_t* launches);
cudaError_t launch_mid_jobs(const DevModel& P, const HermiteW& hw, const MidJob* j, int n, int sms, cudaStream_t st,
                            int64_t* launches);

// One forward step of a grid that does not fit the device at once: src -> dst
// (null: not stored) and its stage states Y2, Y3, Y4 to three states in a row
// (null: not kept).
struct FwdStep {
    const double* src;
    double *dst, *stages;
    const double *E0, *Eh, *E1;
    unsigned* fault;
};
cudaError_t launch_fwd_tile(const DevModel& P, const DevGrid& g, const double* gh, const uint8_t* cells,
                            const FwdStep& r, int sms, cudaStream_t st);

// One backward step likewise: y are the stages' states; row[0] (exact mode:
// row[0 .. 2], as AdjRun's groups) the step's row of partial sums.  segs: per
// row segment of the lattice, whether it holds a source cell.
struct AdjStep {
    const double* zin;
    double* zout;
    const double* y[4];
    double* row[3];
    int nsbx;
    unsigned* fault;
};
cudaError_t launch_adj_tile(bool exact, const DevModel& P, const DevGrid& g, const double* gh, const uint8_t* adj,
                            const uint8_t* segs, const AdjStep& r, int sms, cudaStream_t st);

}  // namespace fkadj
