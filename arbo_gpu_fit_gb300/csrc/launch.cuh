// launch.cuh — programmatic dependent launch, device and host side.
#pragma once
#include <cuda_runtime.h>

namespace arbo {

// Programmatic dependent launch: wait for the previous kernel of the stream (its memory is
// visible afterwards), and let the next kernel of the stream start its prologue early. Both are
// no-ops when the kernels are launched without the programmatic-serialization attribute.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// Launch with programmatic stream serialization: the kernel may start while the previous kernel
// of the stream finishes; it calls griddepcontrol.wait before reading that kernel's results.
template <typename... Args>
inline int launch_pdl(void (*kernel)(Args...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl,
                      Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace arbo
