// Programmatic dependent launch. A kernel launched with programmatic stream serialisation is
// scheduled once every CTA of the one before has called launch_dependents() (or left), and
// waits in wait_previous() for that kernel to complete, with its writes visible, before it
// touches any of them. Without the attribute the wait returns at once.
//
// Such a kernel begins while the launches before it still write, so it reads memory by coherent
// loads only: __ldca, __ldcg or plain ones through pointers that are not const __restrict__
// (of which, as of __ldg, the compiler may make non-coherent loads, valid for what nobody
// writes while the kernel lives, and free to move before the wait).
#pragma once

#include <cuda_runtime.h>

namespace mi {
namespace pdl {

__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// kernel<<<grid, block, smem, st>>>(args...) with programmatic stream serialisation
template <class... Params, class... Args>
cudaError_t launch(void (*kernel)(Params...), dim3 grid, unsigned int block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchAttribute attr[1] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = attr;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<Params>(args)...);
}

}  // namespace pdl
}  // namespace mi
