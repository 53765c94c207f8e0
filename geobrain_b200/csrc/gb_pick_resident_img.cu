// Instantiates the resident forward kernels that write the gradient's imaging
// fields, with the exchange through global memory (warps per tile height as
// in gb_pick_resident.cu).
#include "gb_kernels.h"
#include "gb_resident.cuh"

#include <cuda_runtime.h>

namespace gb {
namespace host {
namespace {

template <int R, int NW, int TZ>
ResidentKernel make(int img)
{
    using G = ResGeo<R, NW, TZ>;
    ResidentKernel k;
    k.fn = img == 2 ? (void *)&resident_fwd_kernel<R, NW, TZ, false, 2> : (void *)&resident_fwd_kernel<R, NW, TZ, false, 1>;
    k.smem = G::SMEM;
    k.threads = G::NTH;
    k.tile_words = (size_t)kResParts * G::PART;
    return k;
}

template <int R>
ResidentKernel pick(int tz, int img)
{
    switch (tz) {
    case 4: return make<R, 4, 4>(img);
    case 8: return make<R, 8, 8>(img);
    case 12: return make<R, 8, 12>(img);
    case 16: return make<R, 16, 16>(img);
    case 24: return make<R, 16, 24>(img);
    case 32: return make<R, 16, 32>(img);
    case 36: return make<R, 12, 36>(img);
    case 40: return make<R, 16, 40>(img);
    default: return ResidentKernel{};
    }
}

}  // namespace

ResidentKernel resident_img_kernel(int R, int tz, int img)
{
    return R == 2 ? pick<2>(tz, img) : R == 4 ? pick<4>(tz, img) : ResidentKernel{};
}

}  // namespace host
}  // namespace gb
