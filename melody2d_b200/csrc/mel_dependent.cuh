// Programmatic dependent launch.
#pragma once
#include <cuda_runtime.h>

namespace mel {
// grid_wait: what the kernels before this one wrote is there from here on (nothing to wait for in an
// ordinary launch); grid_release: the next kernel of the stream may start
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
}  // namespace mel

// launch that may start as soon as the kernel before it in the stream releases it; every kernel
// launched so waits (grid_wait) before it reads or writes what others use
template <class... P, class... A>
static void launch_dependent(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = dim3((unsigned)grid); c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = smem; c.stream = s;
    c.attrs = &a; c.numAttrs = 1;
    cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);      // errors: cudaGetLastError by the caller, as for <<<>>>
}
