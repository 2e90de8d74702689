// Device memory of one adjoint, objective or boundary-flux run, and what is
// kept of it between runs.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <utility>
#include <vector>

#include "dugks_internal.h"

namespace dugks {

// Memory that runs have given back, by device, for the next run of any handle
// there: mapping and unmapping the 950 MB of a 12-step run with 4,096 cells and
// 1,024 DVs takes as long as its kernels.  At most kKeep bytes a device; what is
// oldest goes first.  All of it goes back to the device before an allocation of
// any handle fails (device_malloc), when the device's last handle is destroyed
// and on dugks_release_memory.  Every block in it is idle.  (dugks_abi.cpp)
constexpr size_t kKeep = size_t(2) << 30;
void* take_kept(int device, size_t bytes);
void keep(int device, void* p, size_t bytes);
// cudaMalloc on the current device; no error is left for cudaGetLastError
cudaError_t device_malloc(void** p, size_t bytes);

struct Arena {
    dugks_handle* h;
    std::vector<std::pair<void*, size_t>> p;
    double bytes = 0;
    explicit Arena(dugks_handle* h) : h(h) {}
    Arena(const Arena&) = delete;
    Arena& operator=(const Arena&) = delete;
    ~Arena() {
        // (a run that ended early may have work in flight)
        if (!p.empty()) cudaStreamSynchronize(h->stream);
        for (auto& q : p) keep(h->device, q.first, q.second);
    }
    template <class T>
    int get(dugks_handle* h, T** out, size_t n) {
        const size_t b = std::max<size_t>(n, 1) * sizeof(T);
        void* q = take_kept(h->device, b);
        if (!q) {
            const cudaError_t e = device_malloc(&q, b);
            if (e != cudaSuccess)
                return set_error(h, e == cudaErrorMemoryAllocation ? DUGKS_ERR_OOM : DUGKS_ERR_CUDA,
                                 "dugks_adjoint_run: cudaMalloc of " + std::to_string(b) + " bytes: " +
                                     cudaGetErrorString(e));
        }
        p.emplace_back(q, b);
        bytes += static_cast<double>(b);
        *out = static_cast<T*>(q);
        return DUGKS_OK;
    }
    template <class T>
    int put(dugks_handle* h, T** out, const std::vector<T>& v) {
        if (int st = get(h, out, v.size())) return st;
        if (v.empty()) return DUGKS_OK;
        return check(h, cudaMemcpyAsync(*out, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
    }
    template <class T>
    int zeros(dugks_handle* h, T** out, size_t n) {
        if (int st = get(h, out, n)) return st;
        return check(h, cudaMemsetAsync(*out, 0, std::max<size_t>(n, 1) * sizeof(T), h->stream));
    }
    static int check(dugks_handle* h, cudaError_t e) {
        return e == cudaSuccess ? DUGKS_OK : set_error(h, DUGKS_ERR_CUDA, cudaGetErrorString(e));
    }
};

}  // namespace dugks
