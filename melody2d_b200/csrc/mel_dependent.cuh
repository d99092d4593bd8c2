// Programmatic dependent launch.
#pragma once
#include <cuda_runtime.h>

namespace mel {
// grid_wait: what the kernels before this one wrote is there from here on (nothing to wait for in an
// ordinary launch); grid_release: the next kernel of the stream may start
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class T> __device__ __forceinline__ T ld_l2(const T* p) { return __ldcg(p); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
}  // namespace mel

// Launch that may start as soon as the kernel before it in the stream releases it.  A kernel launched so
// waits (grid_wait) before it reads or writes what others use, with one exception, the body kernel, which
// starts beside the contact pass and reads some of the state that the body kernel before wrote.
// That rests on this invariant: every thread of a kernel waits before it releases (the contact pass, and
// every kernel that may stand between two body kernels), so that what ran before the released kernel's
// predecessor has ended and its writes are in L2 when the successor starts.  Only grid_wait itself
// promises that a thread sees them, though, so what is read before it is read from L2 (ld_l2, or a
// bulk copy), where no line of an L1 cache can be older.  A kernel that releases first (the body kernel)
// must not be followed by one that reads before it waits.
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
