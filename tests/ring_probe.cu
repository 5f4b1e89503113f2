// Test probe (built by tests/test_gpu_ring.py): one CTA fills the ring of the
// middle tile of 3 x 3 from an exchange area given by the host.
#include <cuda_runtime.h>

#include "../adjoint-optimization_b200/csrc/fk_ring.cuh"

using namespace fkadj;

struct S {
    static constexpr int TX = 16, RW = TX + 2 * HALO, TY = 5, PA = (TY + 2 * HALO) * RW;
};
constexpr int NROWS = 3 * S::TY, NCOLS = 3 * S::TX, LD = NCOLS + 2 * HALO, PLANE = (NROWS + 2 * HALO) * LD;

__global__ void __launch_bounds__(96) k_ring_probe(const Tagged* __restrict__ x, int by, int bx, unsigned long long tag,
                                                   double* __restrict__ out, int* __restrict__ status,
                                                   unsigned* __restrict__ fault) {
    __shared__ double A[3 * S::PA];
    __shared__ int2 ring[8 * S::RW + 8 * S::TY];
    for (int q = threadIdx.x; q < 3 * S::PA; q += blockDim.x) A[q] = -1.0;
    const int i0 = by * S::TY, j0 = bx * S::TX;
    const int count = ring_table<S>(ring, LD, S::TY, i0, j0, NROWS, NCOLS);
    __syncthreads();
    const bool ok = read_ring<S, 50000000ull>(A, ring, count, x + i0 * LD + j0, tag, PLANE, fault);
    if (threadIdx.x == 0) *status = ok;
    for (int q = threadIdx.x; q < 3 * S::PA; q += blockDim.x) out[q] = A[q];
}

// h_x: 3 x PLANE values and tags; h_out: 3 windows; fault: before and after.
extern "C" int probe_ring(const void* h_x, int by, int bx, unsigned long long tag, double* h_out, int* h_status,
                          unsigned* h_fault, float* ms) {
    if (by < 0 || by > 2 || bx < 0 || bx > 2) return (int)cudaErrorInvalidValue;
    Tagged* x = nullptr;
    double* out = nullptr;
    int* status = nullptr;
    unsigned* fault = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    const size_t in = 3 * (size_t)PLANE * sizeof(Tagged), ob = 3 * (size_t)S::PA * sizeof(double);
    cudaError_t e = cudaMalloc(&x, in);
    if (!e) e = cudaMalloc(&out, ob);
    if (!e) e = cudaMalloc(&status, sizeof(int));
    if (!e) e = cudaMalloc(&fault, sizeof(unsigned));
    if (!e) e = cudaMemcpy(x, h_x, in, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(fault, h_fault, sizeof(unsigned), cudaMemcpyHostToDevice);
    if (!e) e = cudaEventCreate(&e0);
    if (!e) e = cudaEventCreate(&e1);
    if (!e) e = cudaEventRecord(e0);
    if (!e) {
        k_ring_probe<<<1, 96>>>(x, by, bx, tag, out, status, fault);
        e = cudaGetLastError();
    }
    if (!e) e = cudaEventRecord(e1);
    if (!e) e = cudaEventSynchronize(e1);
    if (!e) e = cudaEventElapsedTime(ms, e0, e1);
    if (!e) e = cudaMemcpy(h_out, out, ob, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(h_status, status, sizeof(int), cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(h_fault, fault, sizeof(unsigned), cudaMemcpyDeviceToHost);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(x);
    cudaFree(out);
    cudaFree(status);
    cudaFree(fault);
    return (int)e;
}
