// Kernels of one stream that follow one another step after step, launched so that the
// next one's blocks are placed while the last blocks of the one before still run
// (programmatic dependent launch).
//
// A chained kernel starts with chain_next(), which lets the kernel after it be placed
// once all its own blocks run, and calls chain_wait() in every thread before its first
// access to global memory: the wait ends when the kernel before it has completed and
// its writes are visible.  Since every chained kernel waits, each one also comes after
// all those before it.  After anything but a kernel the launch is an ordinary one.
#pragma once

#include <cuda_runtime.h>

namespace fdtd {

__device__ __forceinline__ void chain_next() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t launch_chained(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                           const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, args...);
    if (e != cudaSuccess) cudaGetLastError();  // returned, not left for a later launch
    return e;
}

}  // namespace fdtd
