// Launch attributes shared by the host code of every session.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "scene.h"

namespace monki {

// Opt a kernel into kBandMaxBytes of dynamic shared memory beside its static one, once per
// kernel and device. The limit belongs to the kernel, not to a launch, and sessions of other
// scenes launch the same kernel from other threads: set to one scene's own band it would drop
// below what another thread is about to launch with, and that launch fails.
inline cudaError_t allow_band(const void* fn) {
    static std::mutex lock;
    static std::vector<std::pair<const void*, int>> done;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> guard(lock);
    const std::pair<const void*, int> key{fn, device};
    if (std::find(done.begin(), done.end(), key) != done.end()) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBandMaxBytes));
    if (e == cudaSuccess) done.push_back(key);
    return e;
}

}  // namespace monki
