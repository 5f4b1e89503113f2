// Test probe (built by tests/test_gpu_drain.py): windows through a ring of
// three barriers on one CTA, the last of them missed by the wait that counts.
#include <cuda_runtime.h>

#include "../adjoint-optimization_b200/csrc/fk_bulk.cuh"

using namespace fkadj;

constexpr int WIDTH = 72, ROWS = 4, NT = 64, N = 3, WINDOW = 3 * ROWS * WIDTH;

// Windows 0 .. total - 1 of src (WINDOW doubles each, planes ROWS x WIDTH) in
// turn into three buffers; window total - 2 is posted `extra` bytes more than
// its copies deliver.  The last two are left to bulk_drain, then written out.
__global__ void __launch_bounds__(NT) k_drain_probe(const double* __restrict__ src, int total, unsigned extra,
                                                    unsigned long long limit_ns, double* __restrict__ out) {
    __shared__ double4 S4[N * WINDOW / 4];
    __shared__ uint64_t bars[N];
    double* S = reinterpret_cast<double*>(S4);
    const uint32_t bar = bulk_begin(&bars[0]);
    bulk_begin(&bars[1]);
    bulk_begin(&bars[2]);
    __syncthreads();
    for (int j = 0; j < total; ++j) {
        const uint32_t b = bar + 8 * (j % N);
        if (j >= N) {  // the buffer's last window has arrived
            bulk_wait(b, limit_ns, (unsigned)((j - N) / N) & 1u);
            __syncthreads();
        }
        bulk_arrive(b, bulk_bytes<WIDTH>(ROWS) + (j == total - 2 ? extra : 0));
        __syncthreads();
        bulk_issue<ROWS, WIDTH, NT>(b, S + (j % N) * WINDOW, src + (long long)j * WINDOW, WIDTH, ROWS * WIDTH, ROWS);
    }
    bulk_drain<N>(bar, total - 2, total - 1, limit_ns);
    __syncthreads();
    for (int u = 0; u < 2; ++u)
        for (int q = threadIdx.x; q < WINDOW; q += NT) out[u * WINDOW + q] = S[((total - 2 + u) % N) * WINDOW + q];
}

extern "C" int probe_drain(const double* h_src, int total, unsigned extra, unsigned long long limit_ns, double* h_out,
                           float* ms) {
    if (total < 2 || total > 64) return (int)cudaErrorInvalidValue;
    double *d_src = nullptr, *d_out = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    const size_t in = sizeof(double) * WINDOW * (size_t)total, out = sizeof(double) * WINDOW * 2;
    cudaError_t e = cudaMalloc(&d_src, in);
    if (!e) e = cudaMalloc(&d_out, out);
    if (!e) e = cudaMemcpy(d_src, h_src, in, cudaMemcpyHostToDevice);
    if (!e) e = cudaEventCreate(&e0);
    if (!e) e = cudaEventCreate(&e1);
    if (!e) e = cudaEventRecord(e0);
    if (!e) {
        k_drain_probe<<<1, NT>>>(d_src, total, extra, limit_ns, d_out);
        e = cudaGetLastError();
    }
    if (!e) e = cudaEventRecord(e1);
    if (!e) e = cudaEventSynchronize(e1);
    if (!e) e = cudaEventElapsedTime(ms, e0, e1);
    if (!e) e = cudaMemcpy(h_out, d_out, out, cudaMemcpyDeviceToHost);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(d_src);
    cudaFree(d_out);
    return (int)e;
}
