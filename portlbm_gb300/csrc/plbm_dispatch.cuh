// plbm_dispatch.cuh — maps runtime (precision, layout) to a template instantiation.
#pragma once
#include "plbm_dependent.cuh"
#include "plbm_kernels.cuh"

namespace plbm {
// Launches a step kernel (one that calls step_begin) with programmatic stream serialization.
inline cudaError_t launch_step_kernel(void (*kernel)(StepParams), dim3 grid, dim3 block, cudaStream_t s, const StepParams &p)
{
    return launch_dependent(kernel, grid, block, 0, s, p);
}
}  // namespace plbm

#define PLBM_CASE(KER, PR, LA) case (PR) * 3 + (LA): return launch_step_kernel(KER<PR, LA>, grid, block, s, p);
#define PLBM_ALL_CASES(KER) PLBM_ALL_CASES_2(KER, KER)
// BOUND: the kernel of the F64_STRICT, F64_PLAIN and F64_Q60 forms
#define PLBM_ALL_CASES_2(BOUND, KER)                                                          \
    PLBM_CASE(BOUND, 0, 0) PLBM_CASE(BOUND, 0, 1) PLBM_CASE(BOUND, 0, 2)                       \
    PLBM_CASE(KER, 1, 0) PLBM_CASE(KER, 1, 1) PLBM_CASE(KER, 1, 2)                             \
    PLBM_CASE(KER, 2, 0) PLBM_CASE(KER, 2, 1) PLBM_CASE(KER, 2, 2)                             \
    PLBM_CASE(KER, 3, 0) PLBM_CASE(KER, 3, 1) PLBM_CASE(KER, 3, 2)                             \
    PLBM_CASE(KER, 4, 0) PLBM_CASE(KER, 4, 1) PLBM_CASE(KER, 4, 2)                             \
    PLBM_CASE(KER, 5, 0) PLBM_CASE(KER, 5, 1) PLBM_CASE(KER, 5, 2)                             \
    PLBM_CASE(BOUND, 6, 0) PLBM_CASE(BOUND, 6, 1) PLBM_CASE(BOUND, 6, 2)                       \
    PLBM_CASE(KER, 7, 0) PLBM_CASE(KER, 7, 1) PLBM_CASE(KER, 7, 2)                             \
    PLBM_CASE(BOUND, 8, 0) PLBM_CASE(BOUND, 8, 1) PLBM_CASE(BOUND, 8, 2)

// The porous gather of the shifted forms (f32, f16s, bf16s, f16c; the unshifted forms have one gather).
#define PLBM_POROUS_CASE(KER, PR, LA) case (PR) * 3 + (LA): return launch_step_kernel(KER<PR, LA, true>, grid, block, s, p);
#define PLBM_POROUS_CASES(KER)                                                                \
    PLBM_POROUS_CASE(KER, 3, 0) PLBM_POROUS_CASE(KER, 3, 1) PLBM_POROUS_CASE(KER, 3, 2)        \
    PLBM_POROUS_CASE(KER, 4, 0) PLBM_POROUS_CASE(KER, 4, 1) PLBM_POROUS_CASE(KER, 4, 2)        \
    PLBM_POROUS_CASE(KER, 5, 0) PLBM_POROUS_CASE(KER, 5, 1) PLBM_POROUS_CASE(KER, 5, 2)        \
    PLBM_POROUS_CASE(KER, 7, 0) PLBM_POROUS_CASE(KER, 7, 1) PLBM_POROUS_CASE(KER, 7, 2)
