// A stand-in for the CUDA runtime on the host, linked with the library's own
// objects (test_host_paths.py): memory is host memory, copies and fills are
// made at once, kernels do nothing but are counted by name.  It serves the
// host paths that only a failing call reaches: a device allocation can be made
// to fail, a cooperative launch to be refused, a kernel to report a fault.
// Every state, table and buffer that a sweep's job names is checked to lie in
// live device memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

// what the headers' device functions name (none of them is called here)
using std::fma, std::isinf, std::isnan, std::min;
extern uint3 threadIdx;
int __double2hiint(double);
int __double2loint(double);
double __hiloint2double(int, int);
int __vimin_s32_relu(int, int);

#include "../adjoint-optimization_b200/csrc/fk_run.h"

namespace {

// (made on first use: kernels register themselves before main)
struct Tables {
    std::recursive_mutex mu;
    std::map<const void*, std::string> names;  // host stub -> kernel
    std::map<uintptr_t, size_t> live;          // device allocations
    std::map<const void*, void*> symbols;
    std::map<std::string, int64_t> launches;
};
Tables& tables() {
    static Tables* t = new Tables;
    return *t;
}
size_t capacity = (size_t)64 << 30, in_use = 0, peak = 0;
int64_t allocations = 0, fail_at = -1, fail_n = 0;  // which allocations fail, counted since that was set
int64_t host_allocations = 0, host_fail_at = -1;
int refuse_cooperative = 0;
std::string fault_kernel;
unsigned fault_bits = 0;
int fault_times = 0;
int64_t bad = 0;                            // spans outside live device memory
std::string first_bad;

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t device_alloc(void** p, size_t b) {
    Lock lk(tables().mu);
    const int64_t k = allocations++;
    if ((fail_at >= 0 && k >= fail_at && k < fail_at + fail_n) || in_use + b > capacity) return cudaErrorMemoryAllocation;
    *p = std::aligned_alloc(256, (b + 255) / 256 * 256);
    std::memset(*p, 0x5a, b);
    tables().live[(uintptr_t)*p] = b;
    in_use += b;
    if (in_use > peak) peak = in_use;
    return cudaSuccess;
}

cudaError_t device_free(void* p) {
    Lock lk(tables().mu);
    if (!p) return cudaSuccess;
    auto it = tables().live.find((uintptr_t)p);
    if (it == tables().live.end()) return cudaErrorInvalidValue;
    in_use -= it->second;
    tables().live.erase(it);
    std::free(p);
    return cudaSuccess;
}

void span(const void* p, size_t bytes, const std::string& what) {
    auto it = tables().live.upper_bound((uintptr_t)p);
    bool ok = it != tables().live.begin();
    if (ok) {
        --it;
        ok = (uintptr_t)p + bytes <= it->first + it->second;
    }
    if (!ok && bad++ == 0) first_bad = what;
}

using namespace fkadj;
struct Check {
    const DevGrid& g;
    std::string kernel;
    size_t state() const { return (size_t)3 * g.plane * sizeof(double); }
    void states(const double* p, long long n, const char* what) {
        if (n > 0) span(p, (size_t)n * state(), kernel + " " + what);
    }
    void table(const void* p, size_t bytes, const char* what) { span(p, bytes, kernel + " " + what); }
    void fault(unsigned* f) {
        table(f, sizeof *f, "fault");
        if (fault_times > 0 && kernel.find(fault_kernel) != std::string::npos) --fault_times, *f |= fault_bits;
    }
    void fwd(const FwdJob& j) {
        const FwdRun& r = j.r;
        states(r.src, 1, "src");
        states(r.last, 1, "last");
        if (r.out && r.n - 1 >= r.first) states(r.out, (r.n - 1 - r.first) / r.every + 1, "out");
        if (r.stages) states(r.stages, 3LL * r.n, "stages");
        table(r.Et, sizeof(double) * (r.n + 1), "Et");
        table(r.Eh, sizeof(double) * r.n, "Eh");
        table(r.exchange, run_exchange_bytes(g), "exchange");
        fault(r.fault);
    }
    void adj(const AdjJob& j, bool exact) {
        const AdjRun& r = j.r;
        states(r.zin, 1, "zin");
        states(r.zout, 1, "zout");
        states(r.y_hi, 1, "y_hi");
        states(r.y_lo, 1, "y_lo");
        states(r.y_mid, r.n - 1, "y_mid");
        for (int k = 0; k < r.n; ++k) states(r.pts + (long long)k * r.pts_step * r.stride, exact ? 3 : 1, "pts");
        if (r.nsb < (long long)r.nsbx * g.nrows && bad++ == 0) first_bad = kernel + " rows of partial sums";
        table(r.partial, sizeof(double) * (exact ? 3 : 1) * r.window * r.nsb, "partial");
        table(r.exchange, run_exchange_bytes(g), "exchange");
        fault(r.fault);
    }
    void mid(const MidJob& j) {
        const MidRun& r = j.r;
        states(r.y_hi, 1, "y_hi");
        states(r.y_lo, 1, "y_lo");
        states(r.y_mid, r.n - 1, "y_mid");
        states(r.yh, r.n, "yh");
        table(r.Et - r.n, sizeof(double) * (r.n + 1), "Et");
        table(r.E3 - (r.n - 1), sizeof(double) * r.n, "E3");
        fault(r.fault);
    }
};

// as RunJobs in fk_run.cu
template <class Job>
struct Jobs {
    int n;
    Job job[16];
};

void launched(const void* stub, void** args) {
    Lock lk(tables().mu);
    const std::string k = tables().names[stub];
    ++tables().launches[k];
    auto is = [&](const char* s) { return k.find(s) != std::string::npos; };
    const bool exact = is("ELb1E");
    if (is("k_fwd_run")) {
        auto& j = *static_cast<const FwdJob*>(args[1]);
        Check{j.g, k}.fwd(j);
    } else if (is("k_fwd_jobs")) {
        auto& l = *static_cast<const Jobs<FwdJob>*>(args[1]);
        for (int q = 0; q < l.n; ++q) Check{l.job[q].g, k}.fwd(l.job[q]);
    } else if (is("k_adj_run")) {
        auto& j = *static_cast<const AdjJob*>(args[1]);
        Check{j.g, k}.adj(j, exact);
    } else if (is("k_adj_jobs")) {
        auto& l = *static_cast<const Jobs<AdjJob>*>(args[1]);
        for (int q = 0; q < l.n; ++q) Check{l.job[q].g, k}.adj(l.job[q], exact);
    } else if (is("k_mid_run")) {
        auto& j = *static_cast<const MidJob*>(args[2]);
        Check{j.g, k}.mid(j);
    } else if (is("k_mid_jobs")) {
        auto& l = *static_cast<const Jobs<MidJob>*>(args[2]);
        for (int q = 0; q < l.n; ++q) Check{l.job[q].g, k}.mid(l.job[q]);
    } else if (is("k_fwd_tile")) {
        Check c{*static_cast<const DevGrid*>(args[1]), k};
        auto& r = *static_cast<const FwdStep*>(args[4]);
        c.states(r.src, 1, "src");
        if (r.dst) c.states(r.dst, 1, "dst");
        if (r.stages) c.states(r.stages, 3, "stages");
        c.fault(r.fault);
    } else if (is("k_adj_tile")) {
        Check c{*static_cast<const DevGrid*>(args[1]), k};
        auto& r = *static_cast<const AdjStep*>(args[5]);
        c.states(r.zin, 1, "zin");
        c.states(r.zout, 1, "zout");
        for (int s = 0; s < 4; ++s) c.states(r.y[s], 1, "y");
        c.fault(r.fault);
    }
}

}  // namespace

extern "C" {

// ------------------------------------------------------------ the test's side
void fake_reset(int64_t bytes) {
    Lock lk(tables().mu);
    capacity = bytes > 0 ? (size_t)bytes : (size_t)64 << 30;
    fail_at = -1;
    allocations = 0;
    peak = in_use;
    host_fail_at = -1;
    refuse_cooperative = fault_times = 0;
    bad = 0;
    first_bad.clear();
    tables().launches.clear();
}
void fake_fail_allocations(int64_t k, int64_t n) {
    Lock lk(tables().mu);
    allocations = 0;
    fail_at = k;
    fail_n = n;
}
void fake_fail_host_allocation(int64_t k) { Lock lk(tables().mu); host_allocations = 0; host_fail_at = k; }
int64_t fake_allocations() { Lock lk(tables().mu); return allocations; }
int64_t fake_in_use() { Lock lk(tables().mu); return (int64_t)in_use; }
int64_t fake_peak() { Lock lk(tables().mu); return (int64_t)peak; }
void fake_refuse_cooperative(int on) { Lock lk(tables().mu); refuse_cooperative = on; }
void fake_fault(const char* kernel, unsigned bits, int times) {
    Lock lk(tables().mu);
    fault_kernel = kernel;
    fault_bits = bits;
    fault_times = times;
}
int64_t fake_launches(const char* kernel) {
    Lock lk(tables().mu);
    int64_t n = 0;
    for (auto& l : tables().launches)
        if (l.first.find(kernel) != std::string::npos) n += l.second;
    return n;
}
int64_t fake_bad_spans() { Lock lk(tables().mu); return bad; }
const char* fake_first_bad() { return first_bad.c_str(); }

// ------------------------------------------------------------------- runtime
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, void*, void*, void*, void*, int*) {
    Lock lk(tables().mu);
    tables().names[stub] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

static thread_local struct {
    dim3 grid, block;
    size_t smem;
    void* st;
} pushed;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
    pushed = {grid, block, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
    *grid = pushed.grid;
    *block = pushed.block;
    *smem = pushed.smem;
    *static_cast<void**>(st) = pushed.st;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) {
    launched(f, args);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    for (unsigned k = 0; k < c->numAttrs; ++k)
        if (c->attrs[k].id == cudaLaunchAttributeCooperative && c->attrs[k].val.cooperative && refuse_cooperative)
            return cudaErrorCooperativeLaunchTooLarge;
    launched(f, args);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t b) { return device_alloc(p, b); }
cudaError_t cudaFree(void* p) { return device_free(p); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t b, cudaMemPool_t, cudaStream_t) { return device_alloc(p, b); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return device_free(p); }
cudaError_t cudaHostAlloc(void** p, size_t b, unsigned) {
    Lock lk(tables().mu);
    if (host_allocations++ == host_fail_at) return cudaErrorMemoryAllocation;
    return (*p = std::malloc(b)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMallocHost(void** p, size_t b) { return cudaHostAlloc(p, b, 0); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* fr, size_t* tot) {
    Lock lk(tables().mu);
    *tot = capacity;
    *fr = capacity > in_use ? capacity - in_use : 0;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) { *(uint64_t*)v = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t b, cudaMemcpyKind, cudaStream_t) {
    if (b && (!d || !s)) return cudaErrorInvalidValue;
    if (b) std::memcpy(d, s, b);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t b, cudaStream_t) {
    if (b && !d) return cudaErrorInvalidValue;
    if (b) std::memset(d, v, b);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
    Lock lk(tables().mu);
    if (!tables().symbols[s]) tables().symbols[s] = std::calloc(1, 1 << 22);
    *p = tables().symbols[s];
    return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrCooperativeLaunch ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "refused"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

}  // extern "C"
