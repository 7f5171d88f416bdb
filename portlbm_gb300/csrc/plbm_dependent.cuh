// plbm_dependent.cuh — launches with programmatic stream serialization: the kernel's blocks may start
// while the kernel before it in the stream ends, and wait for it with griddepcontrol.wait.
#pragma once
#include <cuda_runtime.h>

namespace plbm {

// A launch that is refused leaves no error behind for the next cudaGetLastError to find.
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
}

}  // namespace plbm
