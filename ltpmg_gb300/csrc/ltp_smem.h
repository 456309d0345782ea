// ltp_smem.h -- shared-memory limits of kernels, host side.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

namespace ltp {

// Raises a kernel's dynamic shared-memory limit, once per device (the limit is
// the device's own: a process may have contexts on several).  done: the
// devices where it is raised, one word per kernel.
template <typename K>
inline cudaError_t allow_smem(K kernel, size_t bytes, std::atomic<uint64_t> &done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;  // (beyond: raised on every call)
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
    return e;
}

}  // namespace ltp
