// Programmatic dependent launches of the kernels of a time loop.
#pragma once
#include <cuda_runtime.h>

namespace rsgpu {

// Programmatic dependent launch: a kernel launched by launch_pdl may start while the one
// before it in the stream drains.  Before pdl_wait it touches only what no kernel writes
// (descriptors, tables, coefficients); after it everything earlier in the stream is
// complete and visible.  pdl_trigger, always after the wait, lets the next kernel start.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with programmatic stream serialisation (see pdl_wait; the kernel must call it).
template <typename... P, typename... V>
static cudaError_t launch_pdl(void (*k)(P...), dim3 grid, dim3 threads, size_t smem, cudaStream_t st, V... args)
{
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = threads;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

}  // namespace rsgpu
