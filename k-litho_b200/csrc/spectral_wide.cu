// spectral_wide.cu -- the spectral core's grids of 160 to 256 points.
#include "spectral.cuh"

namespace kl {
namespace spec {

int launch_wide(const SpecGeom& g, const float2* band, int nparts, float scale, int nimg, const float2* H,
                const float* lam, int K, int nsets, int nsplit, float2* part, float2* T, unsigned* done,
                cudaStream_t st) {
#define KL_SPEC(RG) return launch<RG, false>(g, band, nparts, scale, nimg, H, lam, K, nsets, nsplit, part, T, done, st)
  switch (g.G) {
    case 160: KL_SPEC(5);
    case 192: KL_SPEC(6);
    case 224: KL_SPEC(7);
    case 256: KL_SPEC(8);
  }
#undef KL_SPEC
  set_error("spec_launch: unsupported spectral grid");
  return KL_ERR_UNSUPPORTED;
}

}  // namespace spec
}  // namespace kl
