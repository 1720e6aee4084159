// socs_rows.cu -- row transforms of the general pipeline for widths with few factors
// of two (socs_gen.cu has those whose pixels split into 64 parts).
//
// A row has a few dozen bins and a thousand pixels, and the register FFTs of
// socs_gen.cu shrink with the power of two in Lx: at odd widths every pixel meets
// every bin, with a twiddle and a coefficient from shared memory each time (1.16 ms for
// 24 images of 2001 x 1203, 1.5 us of HBM traffic each).  These kernels are the
// same sums as register-tiled matrix products:
//   * pixels x and Lx - x share a product (cos even, sin odd in x):
//     sum_b Re(q_b w^{bx}) = C -+ S, C = sum a_b cos, S = sum b_b sin;
//     the row DFT takes u = m[x] + m[Lx-x] against cos and v = m[x] - m[Lx-x] against sin,
//   * a twiddle serves several rows, a coefficient several pixels.
// Twiddles are read from the table of the Lx roots of unity (exact arguments).
#include <algorithm>

#include "kl_device.cuh"
#include "kl_internal.h"
#include "kl_launch.cuh"

namespace kl {

namespace {
constexpr int kT = 256;
constexpr int kW = kT / 32;
constexpr int kSMs = 148;
constexpr int kRows = 64;  // rows of a synthesis tile: 8 warps x 8
constexpr int kX = 64;     // base pixels of a synthesis tile (and their mirrors)

template <typename Kern>
int set_smem(Kern k, size_t bytes) {
  if (bytes > 48 * 1024)
    KL_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return KL_OK;
}
}  // namespace

// out[row][x] = Re sum_b Q[row][b] e^{2 pi i b x/Lx}.  A CTA keeps the twiddles of its 64
// pixels and walks over tiles of 64 rows; a warp has 8 rows x 2 pixels per lane, and
// their mirrors: 64 FMAs per 12 shared loads.
__global__ void __launch_bounds__(kT) k_row_synth(const float2* Q, int nbins, int nrows, int Lx,
                                                  const float2* __restrict__ rlx, float* __restrict__ out) {
  extern __shared__ float4 smem4[];
  const int nbp = (nbins + 1) & ~1;
  float2* w = reinterpret_cast<float2*>(smem4);  // [nbp][64]
  float2* qs = w + (size_t)nbp * kX;             // [64 rows][nbp]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * kX;
  for (int i = tid; i < nbp * kX; i += kT) {
    const int b = i / kX, x = x0 + (i & (kX - 1));
    w[i] = b < nbins ? __ldg(rlx + b * x % Lx) : make_float2(0.f, 0.f);
  }
  if (nbp > nbins)
    for (int i = tid; i < kRows; i += kT) qs[(size_t)i * nbp + nbins] = make_float2(0.f, 0.f);
  dep_wait();
  const int half = Lx / 2;
  for (int r0 = blockIdx.y * kRows; r0 < nrows; r0 += gridDim.y * kRows) {
    const int nr = min(kRows, nrows - r0);
    __syncthreads();
    for (int i = tid; i < kRows * nbins; i += kT) {
      const int r = i / nbins, b = i - r * nbins;
      qs[(size_t)r * nbp + b] = r < nr ? Q[(size_t)r0 * nbins + i] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    float C[8][2], S[8][2];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) C[r][h] = S[r][h] = 0.f;
    const float4* q4 = reinterpret_cast<const float4*>(qs + (size_t)warp * 8 * nbp);
#pragma unroll 2
    for (int b = 0; b < nbp; b += 2) {
      float2 wa[2], wb[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        wa[h] = w[b * kX + lane + 32 * h];
        wb[h] = w[(b + 1) * kX + lane + 32 * h];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 q = q4[(r * nbp + b) >> 1];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          C[r][h] = fmaf(q.x, wa[h].x, fmaf(q.z, wb[h].x, C[r][h]));
          S[r][h] = fmaf(q.y, wa[h].y, fmaf(q.w, wb[h].y, S[r][h]));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = r0 + warp * 8 + r;
      if (row >= nrows) break;
      float* o = out + (size_t)row * Lx;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int x = x0 + lane + 32 * h;
        if (x > half) continue;
        __stcs(o + x, C[r][h] - S[r][h]);
        if (x > 0 && 2 * x != Lx) __stcs(o + Lx - x, C[r][h] + S[r][h]);
      }
    }
  }
  dep_launch();  // the next call's kernel, see kl_launch.cuh
}

// R[row][fx] = sum_x m[row][x] e^{-2 pi i fx x/Lx}, fx < nbins, of the rows of one image
// (blockIdx.y).  A CTA has 16 RPT rows and every bin (F per thread); 32 pixel pairs at a
// time go through shared memory as (u, v), the next ones are loaded meanwhile.  Sums
// of 32 terms are added to the total, so rounding grows with Lx / 64.
// VJP: m is dL/dI of the sigmoid resist, made from the image and its target on the
// way; the loss is added to loss[image].
template <int F, int RPT, bool VJP>
__global__ void __launch_bounds__(kT) k_row_dft(const float* src, int Ly, int Lx, int nbins,
                                                const float2* __restrict__ rlx, const float* targets,
                                                int nsets, float alpha, float thr, double* __restrict__ loss,
                                                float2* __restrict__ R) {
  constexpr int ROWS = 16 * RPT, UP = ROWS + 2, LD = ROWS / kW;  // row pairs (u, v) loaded per thread
  __shared__ __align__(16) float2 U[32][UP];
  __shared__ float2 W[32][16 * F];
  __shared__ double s_loss[kW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
  const int img = blockIdx.y, r0 = blockIdx.x * ROWS, half = Lx / 2;
  const float* m = src + ((size_t)img * Ly + r0) * Lx;
  const float* tg = VJP ? targets + ((size_t)(img / nsets) * Ly + r0) * Lx : nullptr;
  // twiddle table entries of this thread: (x, fx) = (i / 16F, i % 16F), and the step of
  // 32 pixels
  int idx[2 * F], step[2 * F];
#pragma unroll
  for (int k = 0; k < 2 * F; ++k) {
    const int i = tid + kT * k, x = i / (16 * F), fx = i % (16 * F);
    idx[k] = x * fx % Lx;  // (below 32 x 128)
    step[k] = 32 * fx % Lx;
  }
  dep_wait();
  dep_launch();
  float2 a[LD], t[VJP ? LD : 1];
  auto fetch = [&](int x0) {
    const int x = x0 + lane;
#pragma unroll
    for (int k = 0; k < LD; ++k) {
      const int r = warp + kW * k;
      const bool ok = x <= half && r0 + r < Ly, mir = ok && x > 0 && 2 * x != Lx;
      a[k] = make_float2(ok ? m[(size_t)r * Lx + x] : 0.f, mir ? m[(size_t)r * Lx + Lx - x] : 0.f);
      if constexpr (VJP)
        t[k] = make_float2(ok ? tg[(size_t)r * Lx + x] : 0.f, mir ? tg[(size_t)r * Lx + Lx - x] : 0.f);
    }
  };
  float2 acc[RPT][F];
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int f = 0; f < F; ++f) acc[r][f] = make_float2(0.f, 0.f);
  double lsum = 0.0;
  fetch(0);
  for (int x0 = 0; x0 <= half; x0 += 32) {
    float rsum = 0.f;
#pragma unroll
    for (int k = 0; k < LD; ++k) {
      float2 g = a[k];
      if constexpr (VJP) {
        const int x = x0 + lane, r = warp + kW * k;
        const bool ok = x <= half && r0 + r < Ly, mir = ok && x > 0 && 2 * x != Lx;
        auto slope = [&](float I, float target, bool on) {
          const float sg = __frcp_rn(1.0f + __expf(-alpha * (I - thr)));
          const float d = sg - target;
          if (on) rsum = fmaf(d, d, rsum);
          return on ? 2.0f * d * sg * (1.0f - sg) * alpha : 0.f;
        };
        g = make_float2(slope(a[k].x, t[k].x, ok), slope(a[k].y, t[k].y, mir));
      }
      U[lane][warp + kW * k] = make_float2(g.x + g.y, g.x - g.y);
    }
    lsum += (double)rsum;
#pragma unroll
    for (int k = 0; k < 2 * F; ++k) {
      const int i = tid + kT * k;
      W[i / (16 * F)][i % (16 * F)] = __ldg(rlx + idx[k]);
      idx[k] += step[k];
      if (idx[k] >= Lx) idx[k] -= Lx;
    }
    __syncthreads();
    if (x0 + 32 <= half) fetch(x0 + 32);
    float2 c[RPT][F];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int f = 0; f < F; ++f) c[r][f] = make_float2(0.f, 0.f);
#pragma unroll 8
    for (int x = 0; x < 32; ++x) {
      float2 u[RPT], w[F];
#pragma unroll
      for (int r = 0; r < RPT; r += 2) {
        const float4 p = *reinterpret_cast<const float4*>(&U[x][ty * RPT + r]);
        u[r] = make_float2(p.x, p.y);
        u[r + 1] = make_float2(p.z, p.w);
      }
#pragma unroll
      for (int f = 0; f < F; ++f) w[f] = W[x][tx + 16 * f];
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int f = 0; f < F; ++f) {
          c[r][f].x = fmaf(u[r].x, w[f].x, c[r][f].x);
          c[r][f].y = fmaf(u[r].y, w[f].y, c[r][f].y);
        }
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int f = 0; f < F; ++f) acc[r][f] = cadd(acc[r][f], c[r][f]);
    __syncthreads();
  }
  // pixel x = half of even widths has no mirror: u = v there, and sin is 0
  float2* o = R + ((size_t)img * Ly + r0) * nbins;
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int f = 0; f < F; ++f)
      if (r0 + ty * RPT + r < Ly && tx + 16 * f < nbins)
        o[(size_t)(ty * RPT + r) * nbins + tx + 16 * f] = make_float2(acc[r][f].x, -acc[r][f].y);
  if constexpr (VJP) {
    for (int s = 16; s > 0; s >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, s);
    if (lane == 0) s_loss[warp] = lsum;
    __syncthreads();
    if (tid == 0) {
      double sum = 0.0;
      for (int k = 0; k < kW; ++k) sum += s_loss[k];
      atomicAdd(loss + img, sum);
    }
  }
}

int row_synth(const GenGeom& g, const float2* rlx, const float2* Q, int nrows, int nbins, float* out, cudaStream_t st) {
  if (nrows <= 0) return KL_OK;
  const int nbp = (nbins + 1) & ~1, xt = (g.Lx / 2 + kX) / kX, groups = (nrows + kRows - 1) / kRows;
  const size_t sm = sizeof(float2) * (size_t)nbp * (kX + kRows);
  if (int rc = set_smem(k_row_synth, sm)) return rc;
  const int gy = std::max(1, std::min(groups, 4 * kSMs / xt));
  KL_CUDA_TRY(launch_dependent(k_row_synth, dim3(xt, gy), kT, sm, st, Q, nbins, nrows, g.Lx, rlx, out));
  return KL_OK;
}

namespace {
template <int F, int RPT, bool VJP>
int launch_dft(const GenGeom& g, const float2* rlx, const float* src, int nimg, int nbins, const float* targets, int nsets,
               float alpha, float thr, double* loss, float2* R, cudaStream_t st) {
  KL_CUDA_TRY(launch_dependent(k_row_dft<F, RPT, VJP>, dim3((g.Ly + 16 * RPT - 1) / (16 * RPT), nimg), kT, 0, st, src, g.Ly,
                               g.Lx, nbins, rlx, targets, nsets, alpha, thr, loss, R));
  return KL_OK;
}
// 64 rows per CTA read a twiddle half as often as 32, once those fill the SMs thrice
bool wide_tiles(const GenGeom& g, int nimg) { return (long long)nimg * ((g.Ly + 63) / 64) >= 3 * kSMs; }
}  // namespace

int row_dft(const GenGeom& g, const float2* rlx, const float* src, int nimg, int nbins, float2* R, cudaStream_t st) {
  if (nimg <= 0) return KL_OK;
  const bool wide = wide_tiles(g, nimg);
#define KL_DFT(F_)                                                                                              \
  return wide ? launch_dft<F_, 4, false>(g, rlx, src, nimg, nbins, nullptr, 1, 0.f, 0.f, nullptr, R, st)         \
              : launch_dft<F_, 2, false>(g, rlx, src, nimg, nbins, nullptr, 1, 0.f, 0.f, nullptr, R, st)
  switch ((nbins + 15) / 16) {
    case 1: KL_DFT(1);
    case 2: KL_DFT(2);
    case 3: KL_DFT(3);
    case 4: KL_DFT(4);
  }
#undef KL_DFT
  set_error("row_dft: more than 64 bins");
  return KL_ERR_UNSUPPORTED;
}

int row_dft_vjp(const GenGeom& g, const float2* rlx, const float* images, int nimg, int nbins, const float* targets,
                int nsets, float alpha, float thr, double* loss, float2* R, cudaStream_t st) {
  if (nimg <= 0) return KL_OK;
  const bool wide = wide_tiles(g, nimg);
#define KL_DFT(F_)                                                                                              \
  return wide ? launch_dft<F_, 4, true>(g, rlx, images, nimg, nbins, targets, nsets, alpha, thr, loss, R, st)    \
              : launch_dft<F_, 2, true>(g, rlx, images, nimg, nbins, targets, nsets, alpha, thr, loss, R, st)
  switch ((nbins + 15) / 16) {
    case 1: KL_DFT(1);
    case 2: KL_DFT(2);
    case 3: KL_DFT(3);
    case 4: KL_DFT(4);
    case 5: KL_DFT(5);
    case 6: KL_DFT(6);
    case 7: KL_DFT(7);
  }
#undef KL_DFT
  set_error("row_dft_vjp: more than 112 bins");
  return KL_ERR_UNSUPPORTED;
}

}  // namespace kl
