// k_nptl.cu — instantiations of the nptl step kernel (two lattices, 2-D blocks).
#include "plbm_dispatch.cuh"
#include "plbm_launch.h"

namespace plbm {
cudaError_t launch_nptl(int prec, int lay, const StepParams &p, dim3 grid, dim3 block, cudaStream_t s, bool porous,
                        bool vec_rows)
{
    static_assert(VEC_ROW_NODES == 32 * VEC, "a warp's nodes");
    const bool two_byte = vec_rows && (prec == F16S || prec == BF16S || prec == F16C);
    const dim3 vb(32, VEC_ROWS), vg((unsigned)((p.P + 32 * VEC - 1) / (32 * VEC)), (unsigned)((p.H + VEC_ROWS - 1) / VEC_ROWS));
    // 2-byte storage in the stream layout on porous geometries: vectorised rows with the bounce-back
    // merged word-wise
    if (porous && two_byte && lay == STREAM) {
        if (prec == F16S) return launch_step_kernel(k_nptl_vec_porous<F16S>, vg, vb, s, p);
        else if (prec == F16C) return launch_step_kernel(k_nptl_vec_porous<F16C>, vg, vb, s, p);
        else return launch_step_kernel(k_nptl_vec_porous<BF16S>, vg, vb, s, p);
    }
    if (porous && ((prec >= F32 && prec <= BF16S) || prec == F16C)) {
        switch (prec * 3 + lay) {
            PLBM_POROUS_CASES(k_nptl)
        default: return cudaErrorInvalidValue;
        }
    }
    // 2-byte storage in the stream layout: vectorised rows (launch shape of its own)
    if (two_byte && lay == STREAM) {
        if (prec == F16S) return launch_step_kernel(k_nptl_vec<F16S>, vg, vb, s, p);
        else if (prec == F16C) return launch_step_kernel(k_nptl_vec<F16C>, vg, vb, s, p);
        else return launch_step_kernel(k_nptl_vec<BF16S>, vg, vb, s, p);
    }
    switch (prec * 3 + lay) {
        PLBM_ALL_CASES(k_nptl)
    default: return cudaErrorInvalidValue;
    }
}
}  // namespace plbm
