// fdtd_chain.cuh -- launches that overlap with the one before them in their stream (programmatic dependent
// launch): the next kernel's blocks come onto an SM as the last ones of its predecessor leave it, and wait
// there until that has ended and its stores are visible.  Back to back kernels of 8.5 us take 11.2 us a launch
// without it.
#pragma once

#include <cuda_runtime.h>

namespace ptk {

// In a kernel launched by launch_chained, before its first access to memory that another kernel may write:
// lets the next launch come up, and waits for the one before.  Such memory must not be read through the
// non-coherent path (__ldg, __restrict__ const parameters), which the wait does not cover.
__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// chained = false: an ordinary launch (chain_wait returns at once).
template <class... P, class... A>
cudaError_t launch_chained(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool chained, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace ptk
