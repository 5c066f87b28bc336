// Programmatic dependent launch: a kernel launched with launch_after starts while the one before it
// in the stream still runs, sets itself up, and waits (after_previous) until that one has completed
// and its writes are visible before it touches global memory; let_next_start allows the next kernel
// the same.  A predecessor or successor that takes no part in it is ordered as usual.
#pragma once
#include <cuda_runtime.h>

namespace mcw {

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                const A &...args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &attr;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace mcw
