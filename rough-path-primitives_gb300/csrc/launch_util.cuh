// launch_util.cuh -- launch-shape helpers shared by the kernel files.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "ops.hpp"

namespace rpp_gb {

constexpr int kMaxDevices = 64;

// Raise a kernel's dynamic shared-memory ceiling to the device's opt-in maximum
// once per (kernel, device).  The kernel is a template argument so that every
// kernel gets its own flag array, even kernels of identical signature.
template <auto kernel>
inline cudaError_t allow_large_smem(const DeviceInfo& dev) {
    static std::atomic<bool> done[kMaxDevices];
    if (dev.device < 0 || dev.device >= kMaxDevices) return cudaErrorInvalidDevice;
    if (done[dev.device].load(std::memory_order_acquire)) return cudaSuccess;
    // static + dynamic shared memory must fit the opt-in limit
    cudaFuncAttributes attr{};
    cudaError_t err = cudaFuncGetAttributes(&attr, kernel);
    if (err != cudaSuccess) return err;
    const int dynamic_max = dev.max_smem_optin - static_cast<int>(attr.sharedSizeBytes);
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dynamic_max);
    if (err == cudaSuccess) done[dev.device].store(true, std::memory_order_release);
    return err;
}

// CTAs of a launch shape that fit an SM.  The runtime's query takes about as
// long as a small launch, so each host thread remembers its answers (they depend
// on the kernel, the device and the shape alone) in a small direct-mapped table.
template <typename Kernel>
inline cudaError_t ctas_per_sm(Kernel kernel, const DeviceInfo& dev, int threads, size_t smem, int& per_sm) {
    struct Answer {
        const void* kernel;
        size_t smem;
        int device, threads, per_sm;
    };
    static thread_local Answer answers[16] = {};  // (one table per kernel signature)
    const void* key = reinterpret_cast<const void*>(kernel);
    const size_t mixed = (reinterpret_cast<uintptr_t>(key) >> 4) + (smem >> 4) + static_cast<size_t>(threads >> 5);
    Answer& a = answers[mixed % 16];
    if (a.kernel != key || a.smem != smem || a.device != dev.device || a.threads != threads) {
        int n = 0;
        const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
        if (err != cudaSuccess) return err;
        a = Answer{key, smem, dev.device, threads, n};
    }
    per_sm = a.per_sm;
    return cudaSuccess;
}

// Grid for a "one CTA per batch element, grid-stride over the batch" kernel:
// as many CTAs as fit on the device at once, capped by the batch.
template <typename Kernel>
inline cudaError_t batch_grid(Kernel kernel, const DeviceInfo& dev, int threads, size_t smem,
                              int64_t batch, dim3& grid) {
    int per_sm = 0;
    cudaError_t err = ctas_per_sm(kernel, dev, threads, smem, per_sm);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int64_t cap = static_cast<int64_t>(per_sm) * dev.sm_count;
    grid = dim3(static_cast<unsigned>(std::max<int64_t>(1, std::min(batch, cap))));
    return cudaSuccess;
}

// Whether two operand batches share no memory (empty ones share none).
template <typename T>
inline bool apart(const Geometry& g, const TArg<T>& a, const TArg<T>& b, int64_t batch) {
    if (!a.p || !b.p || a.lo > a.hi || b.lo > b.hi) return true;
    auto begin = [&](const TArg<T>& t) { return t.p + g.db[t.lo]; };
    auto end = [&](const TArg<T>& t) { return t.p + (batch - 1) * t.stride + g.db[std::min(t.hi, g.depth) + 1]; };
    return end(a) <= begin(b) || end(b) <= begin(a);
}

// Threads per CTA for a tensor whose largest level has `widest` coefficients.
inline int threads_for(uint32_t widest, int cap = 256) {
    int t = 32;
    while (t < cap && static_cast<uint32_t>(t) < widest) t *= 2;
    return t;
}

}  // namespace rpp_gb
