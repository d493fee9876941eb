// Programmatic dependent launch: a kernel of the evaluation sequence lets the next one
// launch as soon as all of its own blocks have started, and waits for the whole previous
// grid (including its memory operations) before touching anything.  Both instructions
// are no-ops when a kernel was launched without the programmatic attribute.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace nnapgb {

__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The wait alone: the next kernel launches when this one has ended.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with the programmatic-stream-serialization attribute (captured into CUDA graphs
// as a programmatic dependency).
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// Launch after the previous kernel has ended.  A kernel that is let in early starts on an SM
// next to the last blocks of the one before and keeps that SM's split between shared memory
// and L1 for its whole run; a large grid that wants another split is better launched so.
template <typename... KArgs, typename... Args>
cudaError_t launch_after(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace nnapgb
