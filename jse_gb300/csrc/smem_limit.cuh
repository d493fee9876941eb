// Dynamic shared memory beyond 48 KiB.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace nnapgb {

// Lets launches of a kernel take `bytes` of dynamic shared memory on the current device (48 KiB
// need no call).  The attribute belongs to a kernel and a device and is shared by every thread of
// the process, so it only grows, under a lock, and is remembered by both: a second device takes
// its own, and a smaller call of another thread does not lower it before this one's launch.
inline cudaError_t allow_smem(const void* kern, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> raised;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& most = raised[{dev, kern}];
    if (bytes <= most) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) most = bytes;
    return e;
}
template <typename... KArgs>
cudaError_t allow_smem(void (*kern)(KArgs...), size_t bytes) {
    return allow_smem(reinterpret_cast<const void*>(kern), bytes);
}

}  // namespace nnapgb
