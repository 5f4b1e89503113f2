// fk_ring.cuh -- the edge exchange of the sweep kernels (fk_run.cu): the ring
// of cells around a CTA's tile, written by its neighbours and read by itself.
#pragma once

#include "fk_bulk.cuh"
#include "fk_run.h"

namespace fkadj {

// One exchanged value: the state's double and the number of the step it
// belongs to, read and written as one 16-byte access.
struct alignas(16) Tagged {
    double v;
    unsigned long long tag;
};
__device__ __forceinline__ void put_tagged(Tagged* p, double v, unsigned long long tag) {
    asm volatile(
        "{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}" ::"l"(p),
        "l"(__double_as_longlong(v)), "l"(tag)
        : "memory");
}
__device__ __forceinline__ Tagged get_tagged(const Tagged* p) {
    long long v;
    unsigned long long t;
    asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}"
                 : "=l"(v), "=l"(t)
                 : "l"(p)
                 : "memory");
    return {__longlong_as_double(v), t};
}

// The 4-cell ring around the tile, one entry per cell: x = its place in
// window A, y = its offset from the window's origin in a state plane, or -1
// outside the grid's tiles.  Made once a sweep: working the places out at
// every step took 2.5 us of it at 512 x 512.
template <class S>
__device__ __forceinline__ int ring_table(int2* ring, int ld, int rows, int i0, int j0, int nrows, int ncols_tiled) {
    const int count = 8 * S::RW + 8 * rows;
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
        int r, c;
        if (i < 8 * S::RW) {
            r = i / S::RW;
            c = i - r * S::RW;
            if (r >= 4) r += rows;
        } else {
            const int j = i - 8 * S::RW;
            r = 4 + (j >> 3);
            c = (j & 7) + ((j & 4) ? S::TX : 0);
        }
        const int gi = i0 + r - HALO, gj = j0 + c - HALO;
        const bool on = gi >= 0 && gi < nrows && gj >= 0 && gj < ncols_tiled;
        ring[i] = make_int2(r * S::RW + c, on ? r * ld + c : -1);
    }
    return count;
}

// Fills the ring of window A with the values of step `tag` (3 x grid planes of
// Tagged at x, window origin included).  Each thread polls its own cells, the
// six values of two of them in flight until all have arrived (one after the
// other, each would cost its own round trip to L2); ring cells outside the
// grid's tiles are left alone (NaN since the sweep's start).  One outcome for
// the CTA, which ends synchronised: false when a wait expired, after 2 s of
// wall time, or another CTA gave up; *fault is then set and the caller
// returns.  All CTAs are resident (cooperative launch), so only a CTA that
// gave up is ever waited for in vain.
template <class S, uint64_t LIMIT_NS = 2000000000ull>
__device__ __noinline__ bool read_ring(double* A, const int2* ring, int count, const Tagged* x, unsigned long long tag,
                                       long long plane, unsigned* fault) {
    constexpr int N = 2;
    bool ok = true;
    for (int base = threadIdx.x; base < count && ok; base += N * blockDim.x) {
        int2 e[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int i = base + u * blockDim.x;
            e[u] = i < count ? ring[i] : make_int2(0, -1);
        }
        uint64_t t0 = 0;
        bool all = false;
        for (int it = 0; !all && ok; ++it) {
            Tagged got[N][3];
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (e[u].y >= 0) {
#pragma unroll
                    for (int f = 0; f < 3; ++f) got[u][f] = get_tagged(x + f * plane + e[u].y);
                }
            all = true;
#pragma unroll
            for (int u = 0; u < N; ++u)
                if (e[u].y >= 0) {
                    if (got[u][0].tag == tag && got[u][1].tag == tag && got[u][2].tag == tag) {
#pragma unroll
                        for (int f = 0; f < 3; ++f) A[f * S::PA + e[u].x] = got[u][f].v;
                        e[u].y = -1;
                    } else {
                        all = false;
                    }
                }
            if ((it & 255) == 255) {
                const uint64_t now = bulk_now_ns();
                if (!t0) t0 = now;
                unsigned f;
                asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(fault) : "memory");
                ok = now - t0 <= LIMIT_NS && !(f & FAULT_TIMEOUT);
            }
        }
    }
    if (!ok) atomicOr(fault, FAULT_TIMEOUT);
    return !__syncthreads_or(!ok);
}

}  // namespace fkadj
