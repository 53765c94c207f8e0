// Instantiates the adjoint tile step kernels with CPML layers, stencil half-width 2.
#include "gb_adj.cuh"
#include "gb_kernels.h"

#include <cuda_runtime.h>

namespace gb {
namespace host {
namespace {

template <int TZ, int IMGF>
void *pick_f(bool fs, bool rho)
{
    if (fs) return rho ? (void *)&adj_step_kernel<2, TZ, true, true, IMGF, true> : (void *)&adj_step_kernel<2, TZ, true, false, IMGF, true>;
    return rho ? (void *)&adj_step_kernel<2, TZ, false, true, IMGF, true> : (void *)&adj_step_kernel<2, TZ, false, false, IMGF, true>;
}

}  // namespace

// as the damping adjoint: a kernel per imaging format at 16 rows, one that
// reads the format at run time at 32
StepKernel adj_cpml_kernel_r2(int tz, bool fs, bool rho, int img_fmt)
{
    StepKernel k;
    if (tz == 16) {
        k.fn = img_fmt == kImgBF16 ? pick_f<16, kImgBF16>(fs, rho)
             : img_fmt == kImgF24  ? pick_f<16, kImgF24>(fs, rho)
                                   : pick_f<16, kImgF32>(fs, rho);
        k.smem = adj_smem_bytes<2, 16>();
    } else if (tz == 32) {
        k.fn = pick_f<32, -1>(fs, rho);
        k.smem = adj_smem_bytes<2, 32>();
    }
    return k;
}

}  // namespace host
}  // namespace gb
