// k_pair.cu — instantiations of the two-step kernel of nptl and lptl.
#include "plbm_dispatch.cuh"
#include "plbm_launch.h"
#include "plbm_pair.cuh"

namespace plbm {

unsigned two_step_blocks(int W)
{
    static_assert(TWO_STEP_COLUMNS == PAIR_COLUMNS, "a strip's columns");
    const int strips = (W + PAIR_COLUMNS - 1) / PAIR_COLUMNS;
    return (unsigned)((strips + PAIR_WARPS - 1) / PAIR_WARPS);
}

template <int PREC, int L>
static cudaError_t launch(const StepParams &p, int rows, cudaStream_t s)
{
    const dim3 grid(two_step_blocks(p.W), (unsigned)((p.H + rows - 1) / rows));
    return launch_dependent(k_two_steps<PREC, L>, grid, dim3(32, PAIR_WARPS), 0, s, p, rows);
}

#define PLBM_PAIR_CASE(PR, LA) case (PR) * 3 + (LA): return launch<PR, LA>(p, rows, s);
cudaError_t launch_two_steps(int prec, int lay, const StepParams &p, int rows, cudaStream_t s)
{
    switch (prec * 3 + lay) {
        PLBM_PAIR_CASE(F32, 0) PLBM_PAIR_CASE(F32, 1) PLBM_PAIR_CASE(F32, 2)
        PLBM_PAIR_CASE(F16S, 0) PLBM_PAIR_CASE(F16S, 1) PLBM_PAIR_CASE(F16S, 2)
        PLBM_PAIR_CASE(BF16S, 0) PLBM_PAIR_CASE(BF16S, 1) PLBM_PAIR_CASE(BF16S, 2)
        PLBM_PAIR_CASE(F16C, 0) PLBM_PAIR_CASE(F16C, 1) PLBM_PAIR_CASE(F16C, 2)
        PLBM_PAIR_CASE(F64_Q60, 0) PLBM_PAIR_CASE(F64_Q60, 1) PLBM_PAIR_CASE(F64_Q60, 2)
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace plbm
