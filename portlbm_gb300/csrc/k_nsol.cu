// k_nsol.cu — instantiations of the nsol step kernels (one lattice, in-place AA swap).
#include "plbm_dispatch.cuh"
#include "plbm_launch.h"

namespace plbm {
cudaError_t launch_nsol(int prec, int lay, const StepParams &p, unsigned t, dim3 grid, dim3 block, cudaStream_t s)
{
    if ((t & 1u) == 0) {
        if (lay == COLLISION && block.x == 32 && block.y >= 1 && block.y <= (unsigned)NSOL_STAGE_ROWS) {
            switch (prec) {   // the record layout's even step with its stores staged per block
            case 0: return launch_step_kernel(k_nsol_even_staged<0>, grid, block, s, p);
            case 1: return launch_step_kernel(k_nsol_even_staged<1>, grid, block, s, p);
            case 2: return launch_step_kernel(k_nsol_even_staged<2>, grid, block, s, p);
            case 3: return launch_step_kernel(k_nsol_even_staged<3>, grid, block, s, p);
            case 4: return launch_step_kernel(k_nsol_even_staged<4>, grid, block, s, p);
            case 5: return launch_step_kernel(k_nsol_even_staged<5>, grid, block, s, p);
            case 6: return launch_step_kernel(k_nsol_even_staged<6>, grid, block, s, p);
            case 7: return launch_step_kernel(k_nsol_even_staged<7>, grid, block, s, p);
            case 8: return launch_step_kernel(k_nsol_even_staged<8>, grid, block, s, p);
            default: return cudaErrorInvalidValue;
            }
        }
        switch (prec * 3 + lay) {
            PLBM_ALL_CASES_2(k_nsol_even_bound, k_nsol_even)
        default: return cudaErrorInvalidValue;
        }
    } else {
        switch (prec * 3 + lay) {
            PLBM_ALL_CASES_2(k_nsol_odd_bound, k_nsol_odd)
        default: return cudaErrorInvalidValue;
        }
    }
}
}  // namespace plbm
