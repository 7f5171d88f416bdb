// plbm_nn_launch.cuh — programmatic dependent launches of the operator's forward kernels.
#pragma once
#include <cuda_runtime.h>

#include "plbm_dependent.cuh"

// The kernel's launch latency and set-up (barriers, tensor memory, descriptors) overlap the end of the
// kernel before it in the stream: everything that reads or writes activations or parameters comes
// after nn_begin, which waits for that kernel and lets the next one in.  Tensor memory is allocated
// before nn_begin, so the next kernel's blocks never hold columns that this kernel still waits for.
// (A 1 x 256^2 inference of 31 launches: 226 -> 215 us as a graph.)
__device__ __forceinline__ void nn_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

template <typename... P, typename... A>
inline cudaError_t nn_launch(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, A... args)
{
    return plbm::launch_dependent(kernel, grid, dim3(block), smem, s, args...);
}
