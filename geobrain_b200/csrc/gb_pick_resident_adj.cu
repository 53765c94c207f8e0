// Instantiates the resident adjoint kernels (gb_resident_adj.cuh; warps per
// tile height as in gb_pick_resident.cu).
#include "gb_kernels.h"
#include "gb_resident_adj.cuh"

#include <cuda_runtime.h>

namespace gb {
namespace host {
namespace {

template <int R, int NW, int TZ>
ResidentKernel make(bool rho)
{
    using G = ResGeo<R, NW, TZ>;
    ResidentKernel k;
    k.fn = rho ? (void *)&resident_adj_kernel<R, NW, TZ, true> : (void *)&resident_adj_kernel<R, NW, TZ, false>;
    k.smem = ResAdjGeo<R, NW, TZ>::SMEM;
    k.threads = G::NTH;
    k.tile_words = (size_t)kResParts * G::PART;
    return k;
}

template <int R>
ResidentKernel pick(int tz, bool rho)
{
    switch (tz) {
    case 4: return make<R, 4, 4>(rho);
    case 8: return make<R, 8, 8>(rho);
    case 12: return make<R, 8, 12>(rho);
    case 16: return make<R, 16, 16>(rho);
    case 24: return make<R, 16, 24>(rho);
    case 32: return make<R, 16, 32>(rho);
    case 36: return make<R, 12, 36>(rho);
    case 40: return make<R, 16, 40>(rho);
    default: return ResidentKernel{};
    }
}

}  // namespace

ResidentKernel resident_adj_kernel_for(int R, int tz, bool rho)
{
    return R == 2 ? pick<2>(tz, rho) : R == 4 ? pick<4>(tz, rho) : ResidentKernel{};
}

}  // namespace host
}  // namespace gb
