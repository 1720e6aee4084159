// spectral.cuh -- the SOCS spectral core: mask band -> sum_k lambda_k |E_k|^2 ->
// its band-limited spectrum T (K-Litho-SOCS/klitho_socs.cpp:196-241 calcSOCS),
// for spectral grids of G = 32 RG points, RG = 1 .. 8 (the smallest that holds
// 4N+1).  The K coherent fields live in registers only.
//
// Decomposition.  A grid point q = RG m + r (m < 32) of a length-G transform of
// x[n] is the 32-point transform over m of the input folded mod 32 after a
// twiddle,
//     E(RG m + r) = sum_j w_32^{j m} sum_{n = j mod 32} x[n] w_G^{n r},
// so one thread can produce 32 outputs of one residue r from one row (or
// column) with no exchange with its neighbours (fft32.cuh).  Only |E|^2 is used,
// so phases that depend on the grid point alone are dropped: the column
// transform counts its rows from 0 instead of -Ny.
//   row warps     thread = (kernel, x residue, band row): H_k . M folded over x,
//                 FFT -> 32 columns of the field's row, to shared memory
//   column warps  thread = (kernel, x residue, y residue, column): the column's
//                 rows folded over y, FFT, lambda |E|^2 onto 32 registers
// The two run at the same time on different kernels (rows in two buffers handed
// over by named barriers); KB kernels are in flight at once so that a CTA has
// about eight column warps.  One CTA holds one x residue of an (image, kernel
// slice), or both of a 64-point grid.  Two residues per thread, which reads
// kernel and band values once for both, was measured slower (41 against 35 us for
// 144 images of 24 kernels at G = 64): twice the code per batch outgrows the
// instruction cache.  For the same reason the column warps' transforms, of the
// kernels and back, are one piece of code.
// The intensity is transformed back the same way (y by 32-point FFTs per
// residue straight from the registers, x by a thread per row) and the y
// residues are combined with their twiddles.  What several CTAs hold of one
// image (x residues, kernel slices) goes through global memory and is summed
// in a fixed order: by the CTA that finishes last when it is little, else by
// k_spec_sum.  No clusters: a GPC holds two clusters of 7 or 8 CTAs, which left
// a quarter of the SMs idle.
//
// Kernel values arrive by cp.async into a ring of each thread's own slots, eight
// values (n = 4q+1 .. 4q+4 and their negatives) at a time, so their L2 latency
// stays off the chain and no barrier is needed for them; the plan keeps the
// kernels in that order (spec_columns), padded with zeros to the grid's largest
// band so that the loops have constant lengths.
#pragma once

#include "spec_common.cuh"

namespace kl {
namespace spec {

constexpr int kLastSum = 16;  // slices of an image that its last CTA adds up itself

template <int RG>
struct SpecCfg {
  static constexpr int G = 32 * RG;
  static constexpr int NB = 16 * RG - 1;           // rows of the largest band
  static constexpr int NQ = 2 * RG;                // groups of four frequencies n > 0
  static constexpr int NR = 16 * RG;               // rows of a padded band
  static constexpr int RC = RG == 2 ? 2 : 1;       // x residues per CTA
  static constexpr int CL = RG / RC;               // CTAs per image and slice
  static constexpr int KB = RG == 1 ? 8 : RG <= 5 ? 2 : 1;  // kernels in flight
  static constexpr int CW = KB * RC * RG;          // column warps
  static constexpr int PW = (KB * RC * NB + 31) / 32;  // row warps
  static constexpr int T = 32 * (CW + PW);
  static constexpr int ROW = 32 * PW;
  static constexpr int RING = RG == 6 || RG == 7 ? 12 : 8;  // groups in flight
};

// shared memory (float2 units): kernel loop, then (over the same space) the
// back transform; then the column twiddles and the G roots of unity
template <int RG>
struct SpecSmem {
  size_t e1, ring, twy, roots, total;
  __host__ __device__ SpecSmem(const SpecGeom& g) {
    using C = SpecCfg<RG>;
    e1 = (size_t)C::RC * (4 * C::NQ + 2) * g.nby;
    ring = e1 + (size_t)2 * C::KB * C::RC * C::NR * kP;
    const size_t loop = ring + (size_t)C::RING * 8 * C::ROW;
    const size_t slots = (size_t)(C::KB - 1) * C::RC * RG * 32 * 32 / 2;  // of floats
    size_t fin = (size_t)C::RC * RG * 17 * kP;
    if (C::KB > 1) fin = fin > slots ? fin : slots;
    twy = loop > fin ? loop : fin;
    twy += twy & 1;
    roots = twy + (size_t)RG * C::NR;
    total = roots + C::G;
  }
};

template <int THREADS>
__device__ __forceinline__ void bar_sync(int id) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(THREADS) : "memory");
}
template <int THREADS>
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(THREADS) : "memory");
}

// a * e^{2 pi i N / G}, a constant
template <int N, int G>
__device__ __forceinline__ float2 mul_root(float2 a) {
  constexpr int n = ((N % G) + G) % G;
  if constexpr (n == 0) {
    return a;
  } else {
    constexpr float c = (float)cx::cos2pi(n, G), s = (float)cx::sin2pi(n, G);
    return make_float2(fmaf(a.x, c, -(a.y * s)), fmaf(a.x, s, a.y * c));
  }
}
template <int G>
struct RootTable64 {
  double c[G], s[G];
  constexpr RootTable64() : c(), s() {
    for (int k = 0; k < G; ++k) {
      c[k] = cx::cos2pi(k, G);
      s[k] = cx::sin2pi(k, G);
    }
  }
};
template <int G>
__device__ const RootTable64<G> g_roots64 = RootTable64<G>();

// T(a, b), moved one pixel on odd periods as the reference's shifts do
__device__ __forceinline__ void put_T(const SpecGeom& g, float2* __restrict__ T, int a, int b, float2 s) {
  if (g.dx | g.dy) {
    const float2 ph1 = expi2pi_frac(-(long long)a * g.dy, g.Ly);
    const float2 ph2 = expi2pi_frac(-(long long)b * g.dx, g.Lx);
    s = cmul(s, cmul(ph1, ph2));
  }
  T[(size_t)(a + 2 * g.Ny) * g.ta + (size_t)b * g.tb] = s;
}

// NATURAL: kernels in the kernel layout [k][row][n], read without the ring (for
// callers that cannot hold the other layout).
// part: for grids up to 64 points and several slices [image][slice] spectra; for
// larger grids [image][slice][x residue][4Ny+1][32] sums over the y residues.
template <int RG, bool NATURAL>
__global__ void __launch_bounds__(SpecCfg<RG>::T, 1)
    k_spectral(const float2* band, int nparts, float scale, const SpecGeom g,
               const float2* __restrict__ H, const float* __restrict__ lam, int K, int nsets, int nsplit,
               float2* __restrict__ part, float2* __restrict__ T, unsigned* __restrict__ done) {
  using C = SpecCfg<RG>;
  constexpr int G = C::G, RC = C::RC, CL = C::CL, KB = C::KB, NQ = C::NQ, NR = C::NR, kT = C::T, RING = C::RING;
  constexpr int kFull = 1, kEmpty = 3, kDone = 5, kCols = 6;  // named barriers; two row buffers
  extern __shared__ float4 smem4[];
  __shared__ unsigned s_last;
  float2* sm = reinterpret_cast<float2*>(smem4);
  const SpecSmem<RG> L(g);
  const int nby = g.nby;
  float2* Mh = sm;              // [RC]{[2 NQ][nby][2], [2][nby]}  M(fy, n) w_G^{n c}: n = 1 .. 8 RG in pairs, n = 0
  float2* E1 = sm + L.e1;       // [2][KB][RC][NR][33]
  float2* twy = sm + L.twy;     // [RG][NR] e^{+2 pi i r i/G}
  float2* roots = sm + L.roots; // [G]
  constexpr size_t kE1 = (size_t)KB * RC * NR * kP;
  const size_t kM = (size_t)(4 * NQ + 2) * nby;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int img = blockIdx.x / CL, c0 = (blockIdx.x - img * CL) * RC, split = blockIdx.y;
  const int clip = img / nsets, set = img - clip * nsets;
  const int k0 = (int)(((long long)K * split) / nsplit), k1 = (int)(((long long)K * (split + 1)) / nsplit);
  // last kernel first: kernels come sorted by weight, so the sums stay small until the end
  // (64 kernels at 4096^2: error against 64 bits 3.6e-7 in order, 2.9e-7 in reverse)
  const int nbatch = (k1 - k0 + KB - 1) / KB;

  // row role: kernel slot, x residue and band row
  const int slot1 = tid / (RC * nby), rem1 = tid - slot1 * (RC * nby);
  const int cc1 = rem1 / nby, row1 = rem1 - cc1 * nby;
  const bool rowthr = tid < KB * RC * nby;
  RowFeed<RING, NQ, C::ROW> feed;
  const size_t hs = NATURAL ? (size_t)nby * g.nbx : spec_hstride(g);
  const float2* hk = H;               // the thread's kernel (of batch 0, then the next one)
  int hleft = 0;                      // batches left for it
  float2 h0 = make_float2(0.f, 0.f);  // its value at n = 0
  if (rowthr) {
    hleft = (k1 - k0 - slot1 + KB - 1) / KB;
    if (hleft > 0) {
      hk = H + ((size_t)set * K + (k1 - 1 - slot1)) * hs + (NATURAL ? (size_t)row1 * g.nbx + g.Nx : row1);
      h0 = __ldg(hk);
    }
    if constexpr (!NATURAL) {
      feed.h = hleft > 0 ? hk + spec_n0(g) + row1 : H;
      feed.pair = 2 * nby;
      feed.skip = spec_n0(g) - (ptrdiff_t)((KB + 1) * hs);
      feed.ring = (unsigned)__cvta_generic_to_shared(sm + L.ring + 2 * tid);
      feed.q = feed.put = 0;
      feed.left = hleft;
      feed.bytes = hleft > 0 ? 16 : 0;
#pragma unroll 1
      for (int i = 0; i < RING - 1; ++i) feed.push();
    }
  }

  for (int i = tid; i < G; i += kT) roots[i] = make_float2(g_roots<G>.c[i], g_roots<G>.s[i]);
  if constexpr (RG > 2)
    for (int i = tid; i < RG * NR; i += kT) twy[i] = root_of<G>((i / NR) * (i % NR));
  // padding: zero entries past the band in Mh and E1
  for (int i = tid; i < RC * nby * (4 * NQ - g.Nx); i += kT) {
    const int q = i / nby, cc = q / (4 * NQ - g.Nx), n = g.Nx + 1 + q - cc * (4 * NQ - g.Nx), r = i - q * nby;
    Mh[cc * kM + (size_t)(((n - 1) >> 1) * nby + r) * 2 + ((n - 1) & 1)] = make_float2(0.f, 0.f);
  }
  for (int i = tid; i < 2 * KB * RC * (NR - nby) * kP; i += kT) {
    const int s = i / ((NR - nby) * kP);
    E1[(size_t)(s * NR + nby) * kP + (i - s * (NR - nby) * kP)] = make_float2(0.f, 0.f);
  }
  // band: kAhead parts at a time.  Nothing before this point reads or writes what
  // other kernels of the call touch
  dep_wait();
  dep_launch();
  constexpr int kAhead = 16;
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
  __syncthreads();

  // column role: kernel slot, x residue, y residue (the slowest index, so that
  // each scheduler has both y residues of a 64-point grid)
  const int cw = warp - C::PW;
  const int r2 = cw / (KB * RC), cc2 = cw / KB % RC, slot2 = cw % KB;
  float2* Zs = sm;  // [RC][RG][17][33], after the kernels
  if (warp < C::PW) {
    const float2* mc = Mh + cc1 * kM;
    const float2 m0 = rowthr ? mc[4 * NQ * nby + row1] : make_float2(0.f, 0.f);
    const float4* ring = reinterpret_cast<const float4*>(sm + L.ring) + tid;
    float2* e1w = E1 + (size_t)((slot1 * RC + cc1) * NR + row1) * kP;
    int take = 0;
#pragma unroll 1
    for (int b = 0; b < nbatch; ++b) {
      float2 v[32];
      if (rowthr) {
        v[0] = cmul(h0, m0);
        const float4* mp = reinterpret_cast<const float4*>(mc) + row1;
        const float4* mn = reinterpret_cast<const float4*>(mc) + (nby - 1 - row1);
        // groups n = 4q+1 .. 4q+4: fold index n mod 32, and 32 - (n mod 32) for -n
        static_for<0, NQ>([&](auto q) {
          constexpr int u = 4 * decltype(q)::value;
          float2 h[4], m[4];
          auto pairs = [](float2 (&o)[4], float4 a, float4 b) {
            o[0] = make_float2(a.x, a.y);
            o[1] = make_float2(a.z, a.w);
            o[2] = make_float2(b.x, b.y);
            o[3] = make_float2(b.z, b.w);
          };
          [[maybe_unused]] const float4* s = ring + (size_t)take * 4 * C::ROW;
          if constexpr (!NATURAL) {
            feed.push();  // into the slot taken RING - 1 groups ago
            cp_wait<RING - 1>();
            take = take + 1 == RING ? 0 : take + 1;
          }
          // index j = n mod 32 is reached first by n = j up to 16, by -n = j - 32 above
          if constexpr (NATURAL) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              h[i] = hleft > 0 && u + i + 1 <= g.Nx ? __ldg(hk + (u + i + 1)) : make_float2(0.f, 0.f);
          } else {
            pairs(h, s[0], s[C::ROW]);
          }
          pairs(m, mp[0], mp[nby]);
          static_for<0, 4>([&](auto i) {
            constexpr int n = u + decltype(i)::value + 1, j = n & 31;
            v[j] = n <= 16 ? cmul(h[i], m[i]) : cfma(h[i], m[i], v[j]);
          });
          if constexpr (NATURAL) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              h[i] = hleft > 0 && u + i + 1 <= g.Nx ? __ldg(hk - (u + i + 1)) : make_float2(0.f, 0.f);
          } else {
            pairs(h, s[2 * C::ROW], s[3 * C::ROW]);
          }
          pairs(m, mn[0], mn[nby]);
          static_for<0, 4>([&](auto i) {
            constexpr int n = u + decltype(i)::value + 1, j = (32 - (n & 31)) & 31;
            v[j] = n < 16 ? cmulc(h[i], m[i]) : cfma(h[i], cconj(m[i]), v[j]);
          });
          mp += 2 * nby;
          mn += 2 * nby;
        });
        if constexpr (RG == 1) static_for<9, 24>([&](auto j) { v[j] = make_float2(0.f, 0.f); });
        // the next batch's value at n = 0
        if (--hleft > 0) {
          hk -= (size_t)KB * hs;
          h0 = __ldg(hk);
        } else {
          h0 = make_float2(0.f, 0.f);
        }
        fft32<+1>(v);
      }
      __syncwarp();
      if (b >= 2) bar_sync<kT>(kEmpty + (b & 1));
      if (rowthr) {
        float2* e = e1w + (b & 1) * kE1;
        static_for<0, 32>([&](auto m) { e[m] = v[fft32_pos(decltype(m)::value)]; });
      }
      __threadfence_block();
      __syncwarp();
      bar_arrive<kT>(kFull + (b & 1));
    }
    if (!NATURAL) cp_wait<0>();  // no copy may land in the space that is reused below
    __syncwarp();
    bar_sync<kT>(kDone);
  } else {
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    const float* lams = lam + (size_t)set * K + k0;
    const float2* e1r = E1 + (size_t)(slot2 * RC + cc2) * NR * kP + lane;
    const float4* tw2 = reinterpret_cast<const float4*>(twy + r2 * NR);
    const int ct = tid - C::ROW;  // thread among the column warps
    constexpr int kRows = RC * RG * 17;
    static_assert(kRows <= 32 * C::CW, "one thread per row of the x back transform");
    // batches, then the y and the x back transform (the transform of the other
    // sign: real and imaginary parts swapped before and after)
#pragma unroll 1
    for (int b = 0; b < nbatch + 2; ++b) {
      float lk = 0.f;
      float2 v[32];
      if (b < nbatch) {
        const int k2 = b * KB + slot2;
        if (k2 < k1 - k0) lk = __ldg(lams + (k1 - k0 - 1 - k2));
        bar_sync<kT>(kFull + (b & 1));
        const float2* e = e1r + (b & 1) * kE1;
        if constexpr (RG <= 2) {
          static_for<0, 32>([&](auto i) { v[i] = decltype(i)::value < NR ? e[i * kP] : make_float2(0.f, 0.f); });
          if (r2 == 1) static_for<1, 32>([&](auto i) { v[i] = mul_root<decltype(i)::value, G>(v[i]); });
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
        if (b + 2 < nbatch) bar_arrive<kT>(kEmpty + (b & 1));
      } else if (b == nbatch) {
        bar_sync<kT>(kDone);  // the space of the kernels and rows is free
        if constexpr (KB > 1) {  // the kernel slots' intensities added up
          float* Is = reinterpret_cast<float*>(sm);  // [KB - 1][RC RG][32][32]
          if (slot2 > 0) {
            float* w = Is + ((size_t)(slot2 - 1) * RC * RG + cc2 * RG + r2) * 1024 + lane;
#pragma unroll
            for (int i = 0; i < 32; ++i) w[i * 32] = acc[i];
          }
          bar_sync<C::CW * 32>(kCols);
          if (slot2 == 0) {
#pragma unroll 1
            for (int s = 1; s < KB; ++s) {
              const float* w = Is + ((size_t)(s - 1) * RC * RG + cc2 * RG + r2) * 1024 + lane;
#pragma unroll
              for (int i = 0; i < 32; ++i) acc[i] += w[i * 32];
            }
          }
          bar_sync<C::CW * 32>(kCols);
        }
        static_for<0, 32>([&](auto m) { v[m] = make_float2(0.f, acc[fft32_pos(decltype(m)::value)]); });
      } else {
        // a thread per (x residue, y residue, term) row
        bar_sync<C::CW * 32>(kCols);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float2 x = ct < kRows ? Zs[(size_t)ct * kP + j] : make_float2(0.f, 0.f);
          v[j] = make_float2(x.y, x.x);
        }
      }
      fft32<+1>(v);
      if (b < nbatch) {
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = fmaf(lk, cabs2(v[i]), acc[i]);
      } else if (b == nbatch) {
        // a real column: its terms 17 .. 31 are conjugates
        if (slot2 == 0) {
          float2* z = Zs + (size_t)(cc2 * RG + r2) * 17 * kP + lane;
          static_for<0, 17>([&](auto a) {
            constexpr int p = fft32_pos(decltype(a)::value);
            z[a * kP] = make_float2(v[p].y, v[p].x);
          });
        }
      } else if (ct < kRows) {
        static_for<0, 32>([&](auto m) {
          constexpr int p = fft32_pos(decltype(m)::value);
          Zs[(size_t)ct * kP + m] = make_float2(v[p].y, v[p].x);
        });
      }
    }
  }
  __syncthreads();

  // sum over the y residues of w_G^{-a r} F_r(a mod 32, beta), F_r(-a) = conj F_r(a)(-beta)
  const int A = 2 * g.Ny;
  auto ysum = [&](int cc, int a, int beta) {
    const int al = a & 31;
    const bool cj = al > 16;
    const float2* f = Zs + (size_t)cc * RG * 17 * kP + (cj ? (32 - al) * kP + ((32 - beta) & 31) : al * kP + beta);
    float2 s = make_float2(0.f, 0.f);
    int m = 0;  // a r mod G
    const int am = a < 0 ? a + G : a;
#pragma unroll
    for (int r = 0; r < RG; ++r) {
      float2 x = f[(size_t)r * 17 * kP];
      if (cj) x.y = -x.y;
      s = r == 0 ? x : cfma(x, cconj(roots[m]), s);
      m += am;
      if (m >= G) m -= G;
    }
    return s;
  };
  if constexpr (RG > 2) {
    float2* U = part + (((size_t)img * nsplit + split) * RG + c0) * g.nty * 32;
    for (int i = tid; i < g.nty * 32; i += kT) U[i] = ysum(0, (i >> 5) - A, i & 31);
    return;
  }
  const size_t tsz = (size_t)g.nty * g.ntx;
  float2* To = nsplit > 1 ? part + ((size_t)img * nsplit + split) * tsz : T + (size_t)img * tsz;
  for (int i = tid; i < (int)tsz; i += kT) {
    const int a = i / g.ntx - A, b = i % g.ntx;
    float2 s = ysum(0, a, b & 31);
    if constexpr (RC == 2) s = cfma(ysum(1, a, b & 31), cconj(roots[b]), s);  // b < G
    put_T(g, To, a, b, cscale(s, 1.0f / ((float)g.G * (float)g.G)));
  }
  if (nsplit > 1 && nsplit <= kLastSum) {
    // the CTA that finishes last adds the image's slices, the largest kernels' last
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(done + img, 1u) == (unsigned)nsplit - 1;
    __syncthreads();
    if (s_last) {
      __threadfence();
      const float2* p0 = part + (size_t)img * nsplit * tsz;
      for (int i = tid; i < (int)tsz; i += kT) {
        float2 v = __ldcg(p0 + (nsplit - 1) * tsz + i);
#pragma unroll 8
        for (int s = nsplit - 2; s >= 0; --s) v = cadd(v, __ldcg(p0 + s * tsz + i));
        T[(size_t)img * tsz + i] = v;
      }
      if (tid == 0) done[img] = 0;  // ready for the next launch
    }
  }
}

// T(a, b) of each image: its slices' spectra added up (up to 64 points), or
// sum_c w_G^{-b c} of the slices' x residues
template <int RG>
__global__ void __launch_bounds__(256) k_spec_sum(const float2* part, const SpecGeom g, int nsplit,
                                                  float2* __restrict__ T) {
  constexpr int G = 32 * RG;
  const int tsz = g.nty * g.ntx, i = blockIdx.y * 256 + threadIdx.x, img = blockIdx.x;
  dep_wait();
  dep_launch();
  if (i >= tsz) return;
  float2* Ti = T + (size_t)img * tsz;
  if constexpr (RG <= 2) {
    const float2* p0 = part + (size_t)img * nsplit * tsz + i;
    // in eight chains: in one, 58 slices of equal weight put the image 2.45e-7 from 64
    // bits, now 2.26e-7
    float2 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = make_float2(0.f, 0.f);
    int s = nsplit - 1;
#pragma unroll 2
    for (; s >= 7; s -= 8)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = cadd(v[j], p0[(size_t)(s - j) * tsz]);
    for (; s >= 0; --s) v[0] = cadd(v[0], p0[(size_t)s * tsz]);
#pragma unroll
    for (int h = 4; h > 0; h >>= 1)
#pragma unroll
      for (int j = 0; j < h; ++j) v[j] = cadd(v[j], v[j + h]);
    Ti[i] = v[0];
  } else {
    const int r = i / g.ntx, b = i - r * g.ntx;
    const size_t res = (size_t)g.nty * 32;
    const float2* p0 = part + (size_t)img * nsplit * RG * res + r * 32 + (b & 31);
    float2 v[RG];
#pragma unroll
    for (int c = 0; c < RG; ++c) v[c] = p0[((nsplit - 1) * RG + c) * res];
    for (int s = nsplit - 2; s >= 0; --s)
#pragma unroll
      for (int c = 0; c < RG; ++c) v[c] = cadd(v[c], p0[(s * RG + c) * res]);
    // In 64 bits: the residues' terms of the mean cancel in the other frequencies, and 1/G^2
    // is not a power of two (20 images of 4096^2, G = 224: 3.0e-7 from 64 bits with this sum
    // in 32, 2.8e-7 now; no time)
    double tx = v[0].x, ty = v[0].y;
#pragma unroll
    for (int c = 1; c < RG; ++c) {
      const int m = b * c % G;
      const double wc = g_roots64<G>.c[m], ws = g_roots64<G>.s[m], x = v[c].x, y = v[c].y;
      tx = fma(x, wc, fma(y, ws, tx));
      ty = fma(y, wc, fma(-x, ws, ty));
    }
    constexpr double inv = 1.0 / (G * G);
    put_T(g, Ti, r - 2 * g.Ny, b, make_float2((float)(tx * inv), (float)(ty * inv)));
  }
}

template <int RG, bool NATURAL>
int launch(const SpecGeom& g, const float2* band, int nparts, float scale, int nimg, const float2* H,
           const float* lam, int K, int nsets, int nsplit, float2* part, float2* T,
                unsigned* done, cudaStream_t st) {
  using C = SpecCfg<RG>;
  auto kern = k_spectral<RG, NATURAL>;
  const size_t sm = sizeof(float2) * SpecSmem<RG>(g).total;
  if (sm > 48 * 1024)
    KL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  KL_CUDA_TRY(launch_dependent(kern, dim3((unsigned)nimg * C::CL, nsplit), C::T, sm, st, band, nparts, scale, g, H, lam, K,
                               nsets, nsplit, part, T, done));
  if (RG > 2 || nsplit > kLastSum)
    KL_CUDA_TRY(launch_dependent(k_spec_sum<RG>, dim3(nimg, (g.nty * g.ntx + 255) / 256), 256, 0, st, part, g, nsplit, T));
  return KL_OK;
}

int launch_wide(const SpecGeom& g, const float2* band, int nparts, float scale, int nimg, const float2* H,
                const float* lam, int K, int nsets, int nsplit, float2* part, float2* T, unsigned* done,
                cudaStream_t st);

}  // namespace spec
}  // namespace kl
