// adjoint_spectral.cu -- the adjoint's spectral core for grids up to 128 points:
//   Gam[f] = sum_k lam_k H_k[f] B_k[f],  B_k[f] = (1/G^2) sum_q conj(e_k(q)) gam(q) e^{2 pi i f.q/G},
//   gam(q) = Re sum_{|g| <= 2N} Gb[g] e^{-2 pi i g.q/G},  Gb = conj of the spectrum of dL/dI
// (the adjoint of K-Litho-SOCS/klitho_socs.cpp:196-241; the fields are recomputed on
// chip).  Shared by both pipelines; socs_gen_vjp.cu has the larger grids.
//
// The transforms are those of spectral.cuh: 32 points per thread, residues mod
// RG = G/32 by twiddles.  Per kernel
//   rows     thread = (x residue, band row): H_k . M folded over x, FFT
//   columns  thread = (x, y residue, column): folded over y, FFT = e_k at 32 points,
//            times gam (32 registers for the whole slice, from k_adjoint_gamma), FFT
//            back
//   back     thread = (x residue, band row): the y residues combined, FFT over x,
//            times H_k onto Gam in shared memory (the thread's own entries)
// Rows of kernel k + 1 and back of kernel k run side by side on the two halves of
// the CTA.  The warp FFTs of the previous kernels spent 20 shuffles per 64 points in
// four passes over padded grids (64 us for 32 images of 24 kernels at G = 64, 136 us for 4
// of 32 at G = 128 on clusters).
#include <algorithm>

#include "spec_common.cuh"

namespace kl {
namespace spec {

constexpr int kHalf = 64;  // threads of the rows, and of the back transform

template <int RG>
struct AdjCfg {
  static constexpr int G = 32 * RG;
  static constexpr int NQ = 2 * RG, NR = 16 * RG;
  static constexpr int RC = RG == 2 ? 2 : 1;  // x residues per CTA
  static constexpr int CL = RG / RC;          // CTAs per image and slice
  static constexpr int KB = RG == 1 ? 4 : 1;  // kernels in flight
  static constexpr int CW = KB * RC * RG;     // warps of the columns
  static constexpr int RING = 3;
  static_assert(KB * RC * (16 * RG - 1) <= kHalf && CW <= 4, "the CTA's 128 threads");
};

template <int RG>
struct AdjSmem {
  size_t e1, z, gacc, ring, twy, roots, total;
  __host__ __device__ AdjSmem(const SpecGeom& g) {
    using C = AdjCfg<RG>;
    e1 = (size_t)C::RC * (4 * C::NQ + 2) * g.nby;
    z = e1 + (size_t)C::KB * C::RC * C::NR * kP;           // [KB][RC][RG][32][33]
    gacc = z + (size_t)C::KB * C::RC * RG * 32 * kP;       // [1 + 8 groups][64]
    ring = gacc + (size_t)(1 + 8 * ((g.Nx + 3) / 4)) * kHalf;
    ring += ring & 1;
    twy = ring + (size_t)2 * C::RING * 8 * kHalf;
    roots = twy + (size_t)RG * C::NR;
    total = roots + C::G;
  }
};

// gam of one image at the grid columns of residue c, a CTA each, for the adjoint
// kernel's column threads: gamma[img][c][r][i][lane], i the transform's output order.
// Once per image instead of once per kernel slice, and out of that kernel's code (it
// took 25 us of a single small clip's adjoint there).  A few CTAs read every partial
// band, so the loads in flight bound it: four images at G = 128 (16 bands of 96 KB each)
// 33 us with 16 float2 per thread, 23 with 32.
template <int RG>
__global__ void __launch_bounds__(512) k_adjoint_gamma(const float2* gband, int gparts, const SpecGeom g,
                                                       float* __restrict__ gamma) {
  constexpr int G = 32 * RG, kT = 512, kAhead = 16, kEach = 2;
  extern __shared__ float4 smem4[];
  float2* Gs = reinterpret_cast<float2*>(smem4);  // [nty][ntx] Gb for gx >= 0; then [nty][33] its rows along x
  __shared__ float2 roots[G];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int img = blockIdx.x / RG, c = blockIdx.x - img * RG;
  const int Nx = g.Nx, nty = g.nty, ntx = g.ntx, A = 2 * g.Ny;
  for (int i = tid; i < G; i += kT) roots[i] = make_float2(g_roots<G>.c[i], g_roots<G>.s[i]);
  dep_wait();
  dep_launch();
  const int per = nty * ntx;
  const float2* p0 = gband + (size_t)img * gparts * per;
  for (int i0 = tid; i0 < per; i0 += kEach * kT) {
    float2 v[kEach];
#pragma unroll
    for (int e = 0; e < kEach; ++e) v[e] = make_float2(0.f, 0.f);
    for (int q0 = 0; q0 < gparts; q0 += kAhead) {
      float2 x[kEach][kAhead];
#pragma unroll
      for (int e = 0; e < kEach; ++e)
#pragma unroll
        for (int p = 0; p < kAhead; ++p)
          x[e][p] = q0 + p < gparts && i0 + e * kT < per ? p0[(size_t)(q0 + p) * per + i0 + e * kT]
                                                         : make_float2(0.f, 0.f);
#pragma unroll
      for (int e = 0; e < kEach; ++e)
#pragma unroll
        for (int p = 0; p < kAhead; ++p) v[e] = cadd(v[e], x[e][p]);
    }
#pragma unroll
    for (int e = 0; e < kEach; ++e) {
      const int i = i0 + e * kT;
      if (i >= per) break;
      float2 w = cconj(v[e]);
      if (g.dx | g.dy) {  // the forward model's one-pixel shift of odd periods
        const int r = i / ntx, gx = i - r * ntx, gy = r - A;
        w = cmul(w, cmul(expi2pi_frac(-(long long)gy * g.dy, g.Ly), expi2pi_frac(-(long long)gx * g.dx, g.Lx)));
      }
      Gs[i] = w;
    }
  }
  __syncthreads();
  // rows: gx = j mod 32, |gx| <= 2Nx; Gb(gy, -gx) = conj Gb(-gy, gx).  At most RG
  // terms on each side of 0 (2Nx < 16 RG), one more for j = 0
  float2 v[32];
  if (tid < nty) {
    const float2* rp = Gs + tid * ntx;
    const float2* rn = Gs + (nty - 1 - tid) * ntx;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      v[j] = make_float2(0.f, 0.f);
#pragma unroll
      for (int t = 0; t < (RG + 1) / 2; ++t) {
        const int gp = j + 32 * t, gn = 32 - j + 32 * t;
        if (gp <= 2 * Nx) v[j] = cfma(rp[gp], cconj(roots[(gp * c) % G]), v[j]);
        if (gn <= 2 * Nx) v[j] = cfma(cconj(rn[gn]), roots[(gn * c) % G], v[j]);
      }
    }
    fft32<-1>(v);
  }
  __syncthreads();
  if (tid < nty) static_for<0, 32>([&](auto m) { Gs[(size_t)tid * kP + m] = v[fft32_pos(decltype(m)::value)]; });
  __syncthreads();
  if (warp < RG) {
    const int r = warp;
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < RG; ++t)
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int i = 32 * t + j;
        if (i < nty) v[j] = cfma(Gs[(size_t)i * kP + lane], cconj(roots[(i * r) % G]), v[j]);
      }
    fft32<-1>(v);
    // rows were counted from 0 instead of gy = -2Ny
    float* o = gamma + ((size_t)(img * RG + c) * RG + r) * 1024 + lane;
    static_for<0, 32>([&](auto m) {
      constexpr int p = fft32_pos(decltype(m)::value);
      const float2 w = roots[(A * (RG * decltype(m)::value + r)) % G];
      o[p * 32] = v[p].x * w.x - v[p].y * w.y;
    });
  }
}

template <int RG>
__global__ void __launch_bounds__(128, 2)
    k_adjoint_spectral(const float2* band, int nparts, float scale, const float* gamma,
                       const SpecGeom g, const float2* __restrict__ H, const float* __restrict__ lam, int K,
                       int nsets, int nsplit, float2* __restrict__ gam_out) {
  using C = AdjCfg<RG>;
  constexpr int G = C::G, RC = C::RC, CL = C::CL, KB = C::KB, NQ = C::NQ, NR = C::NR, kT = 128, RING = C::RING;
  extern __shared__ float4 smem4[];
  float2* sm = reinterpret_cast<float2*>(smem4);
  const AdjSmem<RG> L(g);
  const int nby = g.nby, nbx = g.nbx, Nx = g.Nx;
  const size_t kM = (size_t)(4 * NQ + 2) * nby;
  float2* Mh = sm;               // [RC]{[2 NQ][nby][2], [2][nby]}
  float2* E1 = sm + L.e1;        // [KB][RC][NR][33]
  float2* Z = sm + L.z;
  float2* Gacc = sm + L.gacc;
  float2* twy = sm + L.twy;      // [RG][NR] e^{+2 pi i r i/G}
  float2* roots = sm + L.roots;  // [G]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int img = blockIdx.x / CL, c0 = (blockIdx.x - img * CL) * RC, split = blockIdx.y;
  const int clip = img / nsets, set = img - clip * nsets;
  const int k0 = (int)(((long long)K * split) / nsplit), k1 = (int)(((long long)K * (split + 1)) / nsplit);
  // last kernel first, as in k_spectral: the smallest weights are added up first
  const int nbatch = (k1 - k0 + KB - 1) / KB;

  // both halves: kernel slot, x residue, band row; each its own feed of the kernel
  const bool back = tid >= kHalf;
  const int t1 = tid & (kHalf - 1);
  const int slot1 = t1 / (RC * nby), rem1 = t1 - slot1 * (RC * nby);
  const int cc1 = rem1 / nby, row1 = rem1 - cc1 * nby;
  const bool rowthr = t1 < KB * RC * nby;
  RowFeed<RING, NQ, kHalf> feed;
  const size_t hs = spec_hstride(g);
  const float2* hk = H;
  int hleft = 0;
  float2 h0 = make_float2(0.f, 0.f);
  float2* myring = sm + L.ring + (back ? (size_t)RING * 8 * kHalf : 0) + 2 * t1;
  if (rowthr) {
    hleft = (k1 - k0 - slot1 + KB - 1) / KB;
    if (hleft > 0) {
      hk = H + ((size_t)set * K + (k1 - 1 - slot1)) * hs + row1;
      h0 = __ldg(hk);
    }
    feed.h = hleft > 0 ? hk + spec_n0(g) + row1 : H;
    feed.pair = 2 * nby;
    feed.skip = spec_n0(g) - (ptrdiff_t)((KB + 1) * hs);
    feed.ring = (unsigned)__cvta_generic_to_shared(myring);
    feed.q = feed.put = 0;
    feed.left = hleft;
    feed.bytes = hleft > 0 ? 16 : 0;
#pragma unroll 1
    for (int i = 0; i < RING - 1; ++i) feed.push();
  }
  for (int i = tid; i < G; i += kT) roots[i] = make_float2(g_roots<G>.c[i], g_roots<G>.s[i]);
  for (int i = tid; i < RG * NR; i += kT) twy[i] = root_of<G>((i / NR) * (i % NR));
  for (int i = tid; i < RC * nby * (4 * NQ - Nx); i += kT) {
    const int q = i / nby, cc = q / (4 * NQ - Nx), n = Nx + 1 + q - cc * (4 * NQ - Nx), r = i - q * nby;
    Mh[cc * kM + (size_t)(((n - 1) >> 1) * nby + r) * 2 + ((n - 1) & 1)] = make_float2(0.f, 0.f);
  }
  dep_wait();
  dep_launch();
  constexpr int kAhead = 16;
  {
    const int per = nby * g.nf;
    const float2* b0 = band + (size_t)clip * nparts * per;
    for (int i = tid; i < per; i += kT) {
      float2 v = make_float2(0.f, 0.f);
      for (int p0 = 0; p0 < nparts; p0 += kAhead) {
        float2 x[kAhead];
#pragma unroll
        for (int p = 0; p < kAhead; ++p)
          x[p] = p0 + p < nparts ? b0[(size_t)(p0 + p) * per + i] : make_float2(0.f, 0.f);
#pragma unroll
        for (int p = 0; p < kAhead; ++p) v = cadd(v, x[p]);
      }
      v = cscale(v, scale);
      const int r = i / g.nf, n = i - r * g.nf;
      const int at = n == 0 ? 4 * NQ * nby + r : (((n - 1) >> 1) * nby + r) * 2 + ((n - 1) & 1);
#pragma unroll
      for (int cc = 0; cc < RC; ++cc) Mh[cc * kM + at] = c0 + cc == 0 ? v : cmul(v, root_of<G>(n * (c0 + cc)));
    }
  }
  const int r2 = warp / (KB * RC), cc2 = warp / KB % RC, slot2 = warp % KB;
  float gam[32];  // at the column thread's points, in the order the transform leaves its outputs
  if (warp < C::CW) {
    const float* gm = gamma + ((size_t)(img * RG + c0 + cc2) * RG + r2) * 1024 + lane;
#pragma unroll
    for (int i = 0; i < 32; ++i) gam[i] = gm[32 * i];
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) gam[i] = 0.f;
  }
  // rows past the band, Gam
  for (int i = tid; i < KB * RC * (NR - nby) * kP; i += kT) {
    const int s = i / ((NR - nby) * kP);
    E1[(size_t)(s * NR + nby) * kP + (i - s * (NR - nby) * kP)] = make_float2(0.f, 0.f);
  }
  for (int i = tid; i < (1 + 8 * ((Nx + 3) / 4)) * kHalf; i += kT) Gacc[i] = make_float2(0.f, 0.f);
  __syncthreads();

  const float invg2 = 1.0f / ((float)G * (float)G);
  const float* lams = lam + (size_t)set * K + k0;
  const float2* mc = Mh + cc1 * kM;
  const float2 m0 = rowthr ? mc[4 * NQ * nby + row1] : make_float2(0.f, 0.f);
  const float4* ring = reinterpret_cast<const float4*>(myring);
  int take = 0;
  auto group = [&](float2 (&hp)[4], float2 (&hn)[4]) {
    feed.push();
    cp_wait<RING - 1>();
    const float4* s = ring + (size_t)take * 4 * kHalf;
    const float4 a = s[0], b = s[kHalf], c = s[2 * kHalf], d = s[3 * kHalf];
    hp[0] = make_float2(a.x, a.y);
    hp[1] = make_float2(a.z, a.w);
    hp[2] = make_float2(b.x, b.y);
    hp[3] = make_float2(b.z, b.w);
    hn[0] = make_float2(c.x, c.y);
    hn[1] = make_float2(c.z, c.w);
    hn[2] = make_float2(d.x, d.y);
    hn[3] = make_float2(d.z, d.w);
    take = take + 1 == RING ? 0 : take + 1;
  };
  auto next_h0 = [&] {
    if (--hleft > 0) {
      hk -= (size_t)KB * hs;
      h0 = __ldg(hk);
    } else {
      h0 = make_float2(0.f, 0.f);
    }
  };

#pragma unroll 1
  for (int b = 0; b <= nbatch; ++b) {
    if (!back) {
      if (rowthr && b < nbatch) {  // rows of batch b
        float2 v[32];
        v[0] = cmul(h0, m0);
        const float4* mp = reinterpret_cast<const float4*>(mc) + row1;
        const float4* mn = reinterpret_cast<const float4*>(mc) + (nby - 1 - row1);
        static_for<0, NQ>([&](auto q) {
          constexpr int u = 4 * decltype(q)::value;
          float2 hp[4], hn[4];
          group(hp, hn);
          const float4 p0 = mp[0], p1 = mp[nby], n0 = mn[0], n1 = mn[nby];
          const float2 m[4] = {make_float2(p0.x, p0.y), make_float2(p0.z, p0.w), make_float2(p1.x, p1.y),
                               make_float2(p1.z, p1.w)};
          const float2 w[4] = {make_float2(n0.x, n0.y), make_float2(n0.z, n0.w), make_float2(n1.x, n1.y),
                               make_float2(n1.z, n1.w)};
          static_for<0, 4>([&](auto i) {
            constexpr int n = u + decltype(i)::value + 1, j = n & 31, jn = (32 - j) & 31;
            v[j] = n <= 16 ? cmul(hp[i], m[i]) : cfma(hp[i], m[i], v[j]);
            v[jn] = n < 16 ? cmulc(hn[i], w[i]) : cfma(hn[i], cconj(w[i]), v[jn]);
          });
          mp += 2 * nby;
          mn += 2 * nby;
        });
        if constexpr (RG == 1) static_for<9, 24>([&](auto j) { v[j] = make_float2(0.f, 0.f); });
        next_h0();
        fft32<+1>(v);
        float2* e = E1 + (size_t)((slot1 * RC + cc1) * NR + row1) * kP;
        static_for<0, 32>([&](auto m) { e[m] = v[fft32_pos(decltype(m)::value)]; });
      }
    } else if (rowthr && b > 0) {  // back transform of batch b - 1
      const int k2 = (b - 1) * KB + slot1;
      const float lk = k2 < k1 - k0 ? __ldg(lams + (k1 - k0 - 1 - k2)) * invg2 : 0.f;
      float2 v[32];
      const float2* z = Z + ((size_t)(slot1 * RC + cc1) * RG * 32 + (row1 & 31)) * kP;
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = z[j];
#pragma unroll
      for (int r = 1; r < RG; ++r) {
        const float2 w = twy[r * NR + row1];
        const float2* zr = z + (size_t)r * 32 * kP;
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = cfma(zr[j], w, v[j]);
      }
      fft32<+1>(v);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = cscale(v[j], lk);
      float2* ga = Gacc + t1;
      ga[0] = cfma(h0, v[0], ga[0]);
      ga += kHalf;
      static_for<0, NQ>([&](auto q) {
        constexpr int u = 4 * decltype(q)::value;
        float2 hp[4], hn[4];
        group(hp, hn);
        if (u < Nx) {
          static_for<0, 4>([&](auto i) {
            constexpr int n = u + decltype(i)::value + 1, j = n & 31, jn = (32 - j) & 31;
            ga[i * kHalf] = cfma(hp[i], v[fft32_pos(j)], ga[i * kHalf]);
            ga[(4 + i) * kHalf] = cfma(hn[i], v[fft32_pos(jn)], ga[(4 + i) * kHalf]);
          });
          ga += 8 * kHalf;
        }
      });
      next_h0();
    }
    __syncthreads();
    if (b < nbatch && warp < C::CW) {
      const float2* e = E1 + (size_t)(slot2 * RC + cc2) * NR * kP + lane;
      const float4* tw2 = reinterpret_cast<const float4*>(twy + r2 * NR);
      float2 v[32];
      if constexpr (RG == 1) {
        static_for<0, 32>([&](auto i) { v[i] = decltype(i)::value < NR ? e[i * kP] : make_float2(0.f, 0.f); });
      } else {
        static_for<0, NR / 4>([&](auto q) {
          constexpr int i0 = 4 * decltype(q)::value, j = i0 & 31;
          const float4 wa = tw2[i0 / 2], wb = tw2[i0 / 2 + 1];
          const float2 w[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y),
                               make_float2(wb.z, wb.w)};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 x = e[(i0 + i) * kP];
            if constexpr (i0 < 32) v[j + i] = cmul(x, w[i]);
            else v[j + i] = cfma(x, w[i], v[j + i]);
          }
        });
      }
      fft32<+1>(v);
      float2 u[32];
      static_for<0, 32>([&](auto m) {
        constexpr int p = fft32_pos(decltype(m)::value);
        u[m] = make_float2(v[p].x * gam[p], -v[p].y * gam[p]);
      });
      fft32<+1>(u);
      float2* z = Z + ((size_t)((slot2 * RC + cc2) * RG + r2) * 32) * kP + lane;
      static_for<0, 32>([&](auto m) { z[m * kP] = u[fft32_pos(decltype(m)::value)]; });
    }
    __syncthreads();
  }
  cp_wait<0>();
  // the CTA's share of Gam: kernel slots and x residues added up
  float2* out = gam_out + (((size_t)img * nsplit + split) * CL + c0 / RC) * nby * nbx;
  for (int i = tid; i < nby * nbx; i += kT) {
    const int r = i / nbx, n = i - r * nbx - Nx, a = n < 0 ? -n : n;
    const int e = n == 0 ? 0 : 1 + 8 * ((a - 1) >> 2) + (n < 0 ? 4 : 0) + ((a - 1) & 3);
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int sl = 0; sl < KB; ++sl)
#pragma unroll
      for (int cc = 0; cc < RC; ++cc)
        s = cfma(Gacc[(size_t)e * kHalf + (sl * RC + cc) * nby + r], root_of<G>(n * (c0 + cc)), s);
    out[i] = s;
  }
}

namespace {
template <int RG>
int launch_adjoint(const SpecGeom& g, const float2* band, int nparts, float scale, const float2* gband, int gparts,
                   int nimg, const float2* H, const float* lam, int K, int nsets, int nsplit, float* gamma, float2* gam,
                   cudaStream_t st) {
  auto kern = k_adjoint_spectral<RG>;
  const size_t sm = sizeof(float2) * AdjSmem<RG>(g).total;
  const size_t smg = sizeof(float2) * (size_t)g.nty * (g.ntx > kP ? g.ntx : kP);
  if (sm > 48 * 1024)
    KL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  if (smg > 40 * 1024)
    KL_CUDA_TRY(cudaFuncSetAttribute(k_adjoint_gamma<RG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smg));
  KL_CUDA_TRY(launch_dependent(k_adjoint_gamma<RG>, dim3((unsigned)nimg * RG), 512, smg, st, gband, gparts, g, gamma));
  KL_CUDA_TRY(launch_dependent(kern, dim3((unsigned)nimg * AdjCfg<RG>::CL, nsplit), 128, sm, st, band, nparts, scale, gamma,
                               g, H, lam, K, nsets, nsplit, gam));
  return KL_OK;
}

// T(a, b) = (conj Gam[a][b] + Gam[-a][-b]) / (Lx Ly) for |a| <= Ny, 0 <= b <= Nx, zero in
// the rest of [-ay, ay] x [0, nb): the half-plane spectrum of dL/dm.  32 loads in flight
// per thread: 32 shares of four images 10 us (31 with 16)
__global__ void __launch_bounds__(128) k_adjoint_grad(const float2* gam, const SpecGeom g, int nparts, int ay,
                                                      int nb, int sa, int sb, float2* __restrict__ T) {
  dep_wait();
  dep_launch();
  const int i = blockIdx.y * 128 + threadIdx.x, rows = 2 * ay + 1, clip = blockIdx.x;
  if (i >= rows * nb) return;
  const int a = i / nb - ay, b = i % nb;
  const size_t nb2 = (size_t)g.nby * g.nbx;
  float2 f1 = make_float2(0.f, 0.f), f2 = f1;
  if (a >= -g.Ny && a <= g.Ny && b <= g.Nx) {
    const float2* p1 = gam + (size_t)clip * nparts * nb2 + (size_t)(a + g.Ny) * g.nbx + (b + g.Nx);
    const float2* p2 = gam + (size_t)clip * nparts * nb2 + (size_t)(g.Ny - a) * g.nbx + (g.Nx - b);
#pragma unroll 16
    for (int p = nparts - 1; p >= 0; --p) {
      f1 = cadd(f1, p1[p * nb2]);
      f2 = cadd(f2, p2[p * nb2]);
    }
  }
  T[(size_t)clip * rows * nb + (size_t)(a + ay) * sa + (size_t)b * sb] =
      cscale(cadd(cconj(f1), f2), 1.0f / ((float)g.Lx * (float)g.Ly));
}
}  // namespace
}  // namespace spec

size_t adjoint_gamma_elems(const SpecGeom& g, int nimg) { return adjoint_core(g) ? (size_t)nimg * g.G * g.G : 0; }
bool adjoint_core(const SpecGeom& g) { return g.G <= 128; }
int adjoint_shares(const SpecGeom& g) { return g.G <= 64 ? 1 : g.G / 32; }

int adjoint_choose_split(const SpecGeom& g, int nimg, int K) {
  // as spec_choose_split: two CTAs per SM up to 64 points, one above; the fixed part
  // (band, gam, the share of Gam) is about three kernels
  const int kb = g.G == 32 ? 4 : 1;
  const long long slots = g.G <= 64 ? 296 : 148, ctas = (long long)nimg * adjoint_shares(g);
  int best = 1;
  double best_t = 1e30;
  const int most = std::min(kAdjointMaxSplit, (K + kb - 1) / kb);
  for (int ns = 1; ns <= most; ++ns) {
    const int batches = ((K + ns - 1) / ns + kb - 1) / kb;
    const long long waves = (ctas * ns + slots - 1) / slots;
    const double t = (double)waves * (3.0 + batches) + 0.05 * ns;
    if (t < best_t * 0.98) {
      best_t = t;
      best = ns;
    }
  }
  return best;
}

int adjoint_launch(const SpecGeom& g, const float2* band, int nparts, float scale, const float2* gband, int gparts,
                   int nimg, const float2* H, const float* lam, int K, int nsets, int nsplit, float* gamma, float2* gam,
                   cudaStream_t st) {
  if (nimg <= 0) return KL_OK;
  switch (g.G) {
    case 32: return spec::launch_adjoint<1>(g, band, nparts, scale, gband, gparts, nimg, H, lam, K, nsets, nsplit, gamma, gam, st);
    case 64: return spec::launch_adjoint<2>(g, band, nparts, scale, gband, gparts, nimg, H, lam, K, nsets, nsplit, gamma, gam, st);
    case 96: return spec::launch_adjoint<3>(g, band, nparts, scale, gband, gparts, nimg, H, lam, K, nsets, nsplit, gamma, gam, st);
    case 128: return spec::launch_adjoint<4>(g, band, nparts, scale, gband, gparts, nimg, H, lam, K, nsets, nsplit, gamma, gam, st);
  }
  set_error("adjoint_launch: unsupported spectral grid");
  return KL_ERR_UNSUPPORTED;
}

int adjoint_gradient(const SpecGeom& g, const float2* gam, int nclips, int nparts, int ay, int nb, int sa, int sb, float2* T,
                     cudaStream_t st) {
  if (nclips <= 0) return KL_OK;
  KL_CUDA_TRY(launch_dependent(spec::k_adjoint_grad, dim3(nclips, ((2 * ay + 1) * nb + 127) / 128), 128, 0, st, gam, g, nparts,
                               ay, nb, sa, sb, T));
  return KL_OK;
}

}  // namespace kl
