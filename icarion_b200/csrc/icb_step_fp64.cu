// icb_step_fp64.cu — FP64 instantiations of the fused step kernel.
// Built with --fmad=false: no FMA contraction, so the collision-free push
// performs the reference's IEEE double operations in the reference's order.
#include "icb_internal.h"
#define ICB_TF_TABLE_UNIT
#include "icb_step_kernel.cuh"
#include "icb_step_dispatch.cuh"

namespace icb {
cudaError_t launch_step_fp64(int integ, int coll, int field, bool mag, const StepParams& p,
                             dim3 grid, dim3 block, cudaStream_t s) {
    return dispatch_step<kPrecFP64, true>(integ, coll, field, mag, p, grid, block, s);
}

cudaError_t launch_tf_table(const StepParams& p, double* tab, double* tseq, uint32_t stride, cudaStream_t s) {
    k_tf_table<<<p.n_ens, 256, 0, s>>>(p, tab, tseq, stride);
    return cudaGetLastError();
}

cudaError_t launch_angle_table(const double2** tab, cudaStream_t s) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_angle_tab);
    if (e != cudaSuccess) return e;
    *tab = static_cast<const double2*>(p);
    k_angle_table<<<kAngles / 256, 256, 0, s>>>();
    return cudaGetLastError();
}

cudaError_t launch_clock_advance(unsigned long long* step, double* t, const double* dt, int n_ens, uint32_t K,
                                 cudaStream_t s) {
    // a launch of few steps needs no more than a warp
    k_clock_advance<<<n_ens, K >= 64u ? 256 : 32, 0, s>>>(step, t, dt, K);
    return cudaGetLastError();
}
}  // namespace icb
