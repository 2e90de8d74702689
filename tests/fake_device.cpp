// A CUDA runtime on the host with two devices of a given memory, and launches
// that compute nothing but what a test asks about: the C ABI's own host code
// (dugks_abi.cpp, dugks_host.cpp) runs on it without a GPU.  A launch on a
// stream of another device than the current one fails, as on a GPU.
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "dugks_arena.h"
#include "dugks_kernels.cuh"

namespace {

struct Block {
    size_t bytes;
    int device;
};
std::mutex lock;
std::map<void*, Block> blocks;
size_t capacity[2] = {size_t(1) << 40, size_t(1) << 40}, used[2];
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
int last_hzero = -1, last_chunks[2], passes = 0;

int device_of(cudaStream_t s) { return *reinterpret_cast<int*>(s); }
// (a launch reports what cudaGetLastError finds, an error before it included)
cudaError_t launch(cudaStream_t s) {
    const cudaError_t e = device_of(s) == current ? last : cudaErrorInvalidResourceHandle;
    return last = cudaSuccess, e;
}

}  // namespace

extern "C" {

void fake_capacity(int device, size_t bytes) { capacity[device] = bytes; }
size_t fake_used(int device) { return used[device]; }
void fake_current(int device) { current = device; }
int fake_device() { return current; }
int fake_last_hzero() { return last_hzero; }
int fake_last_chunks(int faces) { return last_chunks[faces]; }
int fake_passes() { return passes; }
// a run that takes n blocks of these bytes
int fake_run(dugks_handle* h, const size_t* bytes, int n) {
    cudaSetDevice(h->device);
    dugks::Arena ar(h);
    for (int i = 0; i < n; ++i) {
        unsigned char* p;
        if (int st = ar.get(h, &p, bytes[i])) return st;
    }
    return DUGKS_OK;
}

cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> g(lock);
    n = (n + 511) / 512 * 512;
    if (used[current] + n > capacity[current]) return last = cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    blocks[*p] = {n, current};
    used[current] += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> g(lock);
    auto it = blocks.find(p);
    if (it == blocks.end()) return last = cudaErrorInvalidValue;
    used[it->second.device] -= it->second.bytes;
    blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = capacity[current] - used[current];
    *t = capacity[current];
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t i = 0; i < h; ++i) std::memcpy(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return current = d, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = current, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 2, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int device) { return *v = device ? 74 : 148, cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    return last = cudaSuccess, e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(new int(current));
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return delete reinterpret_cast<int*>(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }

// entry points whose kernels are in files not built here
int dugks_adjoint_run(dugks_handle*, const dugks_objective*, double*, double*, double*, double*, dugks_adjoint_stats*) {
    return DUGKS_ERR_UNSUPPORTED;
}
int dugks_objective_run(dugks_handle*, const dugks_objective*, double*, dugks_adjoint_stats*) {
    return DUGKS_ERR_UNSUPPORTED;
}
int dugks_boundary_fluxes(dugks_handle*, double, double*) { return DUGKS_ERR_UNSUPPORTED; }
int64_t dugks_checkpoint_forward_steps(int32_t, int32_t) { return 0; }
int dugks_cell_macros_noalloc(int32_t, int32_t, const double*, const double*, int32_t, const double*, const double*,
                              const dugks_gas*, double, double*, double*, double*, double*, void*, char*, int32_t) {
    return DUGKS_ERR_UNSUPPORTED;
}

}  // extern "C"

namespace dugks {

cudaError_t launch_stage(const StepArgs& a, int, int, cudaStream_t s, int*) {
    last_hzero = a.hzero;
    last_chunks[0] = a.chunks;
    last_chunks[1] = a.chunks_f;
    return launch(s);
}
cudaError_t launch_init(const StepArgs& a, int, cudaStream_t s) {
    const size_t n = static_cast<size_t>(a.dm.nv_loc) * a.dm.pC;
    for (size_t i = 0; i < n; ++i) {
        static_cast<double*>(a.ds.g)[i] = 1.0;
        static_cast<double*>(a.ds.h)[i] = 0.0;
    }
    return launch(s);
}
cudaError_t launch_pass(const StepArgs&, int, int, cudaStream_t s) { return ++passes, launch(s); }
cudaError_t launch_finish(const StepArgs&, bool, cudaStream_t s) { return launch(s); }
cudaError_t configure_kernels(int, int) { return cudaSuccess; }
cudaError_t launch_upwind_bits(const DevMesh&, uint32_t*, unsigned long long*, cudaStream_t s) { return launch(s); }
cudaError_t launch_list_tangential(const DevMesh&, int2*, unsigned long long*, uint2*, unsigned*, cudaStream_t s) {
    return launch(s);
}
cudaError_t launch_sum_chunks(double*, int, size_t, cudaStream_t s) { return launch(s); }
cudaError_t launch_cell_records(const StepArgs&, cudaStream_t s) { return launch(s); }
cudaError_t launch_adapt(const StepArgs&, const double*, double*, double*, double, double, cudaStream_t s) {
    return launch(s);
}
// FP64 states only
cudaError_t launch_state_order(const StepArgs& a, int, bool second, bool get, const int32_t* iperm, double* buf,
                               size_t first, size_t n, cudaStream_t s) {
    double* st = static_cast<double*>(second ? a.ds.h : a.ds.g);
    for (size_t i = first; i < first + n; ++i) {
        const size_t d = i / a.dm.nC, c = iperm[i % a.dm.nC];
        double& x = st[(c / 32 * a.dm.nv_loc + d) * 32 + c % 32];
        if (get) buf[i - first] = x;
        else x = buf[i - first];
    }
    return launch(s);
}

}  // namespace dugks
