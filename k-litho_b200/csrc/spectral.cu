// spectral.cu -- host side of the spectral core (spectral.cuh) and its grids up to
// 128 points; spectral_wide.cu has the larger ones.
#include "spectral.cuh"

#include <algorithm>

namespace kl {

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
namespace {
int spec_grid(int Nx, int Ny) { return (4 * std::max(Nx, Ny) + 1 + 31) / 32 * 32; }
}  // namespace
SpecGeom spec_geometry(const SocsGeom& s) {
  SpecGeom g{};
  g.Nx = s.Nx; g.Ny = s.Ny; g.nbx = s.nbx; g.nby = s.nby; g.nf = s.nf; g.ntx = s.ntx; g.nty = s.nty;
  g.G = spec_grid(s.Nx, s.Ny); g.Lx = s.Lx; g.Ly = s.Ly; g.dx = s.dx; g.dy = s.dy;
  g.ta = s.ntx;
  g.tb = 1;
  return g;
}
SpecGeom spec_geometry(const GenGeom& s) {
  SpecGeom g{};
  g.Nx = s.Nx; g.Ny = s.Ny; g.nbx = s.nbx; g.nby = s.nby; g.nf = s.nf; g.ntx = s.ntx; g.nty = s.nty;
  g.G = spec_grid(s.Nx, s.Ny); g.Lx = s.Lx; g.Ly = s.Ly; g.dx = s.dx; g.dy = s.dy;
  g.ta = 1;
  g.tb = s.nty;
  return g;
}

int spec_choose_split(const SpecGeom& g, int nimg, int K) {
  // The slice count with the least waves x (batches of kernels + fixed part of a
  // CTA, about three batches: band load, back transform, slice sum).  At 32 points a CTA
  // is small and several share an SM: waves count in fractions, of about 100 CTAs since
  // the early start does not spread them evenly, and the sum over slices weighs as much
  // as the fixed part.  With whole waves 12 to 48 kernels of 24 to 48 clips of 256^2 took
  // up to 1.09 of the warp-FFT kernels' time; 32 clips of 24 kernels (3 slices, now 1)
  // 28.3 -> 23.6 us a call.  Over 384 shapes 1.008 of the best count's time in the
  // geometric mean (1.058 with whole waves).
  const int rg = g.G / 32, kb = rg == 1 ? 8 : rg <= 5 ? 2 : 1;
  const long long slots = 148, ctas = (long long)nimg * (rg == 2 ? 1 : rg);
  int best = 1;
  double best_t = 1e30;
  const int most = std::min(kSpecMaxSplit, (K + kb - 1) / kb);
  for (int ns = 1; ns <= most; ++ns) {
    const int batches = ((K + ns - 1) / ns + kb - 1) / kb;
    const double waves = rg == 1 ? std::max(1.0, ctas * ns / 100.0) : (double)((ctas * ns + slots - 1) / slots);
    const double t = waves * (3.0 + batches) + (rg > 1 ? 0.05 * ns : ns > 1 ? 3.0 + 0.4 * ns : 0.4);
    if (t < best_t * 0.98) {
      best_t = t;
      best = ns;
    }
  }
  return best;
}

size_t spec_kernel_elems(const SpecGeom& g) { return spec::spec_hstride(g); }

size_t spec_part_elems(const SpecGeom& g, int nimg, int nsplit) {
  const size_t n = (size_t)nimg * nsplit;
  if (g.G > 64) return n * (g.G / 32) * g.nty * 32;
  return nsplit > 1 ? n * g.nty * g.ntx : 0;
}

namespace {
// kernels [k][row][n] -> the core's layout; zero past Nx
__global__ void k_spec_columns(const float2* __restrict__ H, const SpecGeom g, size_t hs, size_t total,
                               float2* __restrict__ HT) {
  const int nby = g.nby, n0 = spec::spec_n0(g);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t k = i / hs;
    const int e = (int)(i - k * hs);
    int n = 0, r = e;
    if (e >= n0) {
      const int u = e - n0, grp = u / (8 * nby), v = u - grp * 8 * nby, p = v / (2 * nby), w = v - p * 2 * nby;
      r = w >> 1;
      n = 4 * grp + 2 * (p & 1) + (w & 1) + 1;
      if (n > g.Nx) r = nby;
      if (p >= 2) n = -n;
    }
    HT[i] = r < nby ? H[k * nby * g.nbx + (size_t)r * g.nbx + g.Nx + n] : make_float2(0.f, 0.f);
  }
}

__global__ void k_spec_interleave(const float* __restrict__ re, const float* __restrict__ im, size_t n,
                                  float2* __restrict__ H) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    H[i] = make_float2(re[i], im[i]);
}
}  // namespace

int spec_interleave(const float* re, const float* im, size_t n, float2* H, cudaStream_t st) {
  k_spec_interleave<<<(int)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, st>>>(re, im, n, H);
  KL_CUDA_TRY(cudaGetLastError());
  return KL_OK;
}

int spec_columns(const SpecGeom& g, const float2* H, int nk, float2* HT, cudaStream_t st) {
  const size_t hs = spec::spec_hstride(g), total = hs * nk;
  const int blocks = (int)std::min<size_t>((total + 255) / 256, 148 * 16);
  k_spec_columns<<<blocks, 256, 0, st>>>(H, g, hs, total, HT);
  KL_CUDA_TRY(cudaGetLastError());
  return KL_OK;
}

int spec_launch(const SpecGeom& g, const float2* band, int nparts, float scale, int nimg, const float2* H, bool natural,
                const float* lam, int K, int nsets, int nsplit, float2* part, float2* T,
                unsigned* done, cudaStream_t st) {
  if (nimg <= 0) return KL_OK;
#define KL_SPEC(RG)                                                                                            \
  return natural ? spec::launch<RG, true>(g, band, nparts, scale, nimg, H, lam, K, nsets, nsplit, part, T, done, st) \
                 : spec::launch<RG, false>(g, band, nparts, scale, nimg, H, lam, K, nsets, nsplit, part, T, done, st)
  switch (g.G) {
    case 32: KL_SPEC(1);
    case 64: KL_SPEC(2);
    case 96: KL_SPEC(3);
    case 128: KL_SPEC(4);
  }
#undef KL_SPEC
  if (!natural && g.G <= 256)
    return spec::launch_wide(g, band, nparts, scale, nimg, H, lam, K, nsets, nsplit, part, T, done, st);
  set_error("spec_launch: unsupported spectral grid");
  return KL_ERR_UNSUPPORTED;
}

}  // namespace kl
