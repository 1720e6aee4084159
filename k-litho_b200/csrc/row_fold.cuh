// The fold of a row's bins onto the Hermitian half of a length-P spectrum, as
// the row syntheses of periods Lx = P V with P >= 8 run it.
//
// Lane l of a row needs, for the P pixels l + V i, the spectrum
//   X[k] = sum over b = k mod P of Q[b] e^{2 pi i b l / Lx},   k = 0 .. P-1,
// as Y[k] = X[k] + conj X[P-k].  With b = P j + k the twiddle splits into
// w^k = e^{2 pi i k l / Lx} and u^j, u = e^{2 pi i l / V}, and the conjugate
// half has the same w^k:
//   Y[k] = w^k ( sum_j u^j Q[Pj + k] + conj sum_j u^{j+1} Q[Pj + P - k] ).
// So a bin costs half a broadcast load and four multiply-adds (none where
// j = 0 and k <= P/2), and only the P/2 + 1 sums meet a twiddle of their own:
// 33 per-lane loads instead of 128 for 107 bins at P = 64, where the loads of
// one twiddle per bin and lane (two wavefronts each) and their waits bound
// the kernel.  The powers of u come from a table, each exact to one rounding.
#pragma once
#include "kl_device.cuh"
#include "kl_internal.h"

namespace kl {

// [P/2 + 1][Vp] w^k and [Vp] u, Vp = V rounded up to 32
__host__ __device__ inline int row_fold_stride(int V) { return (V + 31) / 32 * 32; }
__host__ __device__ inline size_t row_fold_elems(int P, int V) { return (size_t)(P / 2 + 2) * row_fold_stride(V); }
// in shared memory up to 96 KB (two CTAs per SM), read from the roots of Lx beyond
inline bool row_fold_in_smem(int P, int V) { return row_fold_elems(P, V) * sizeof(float2) <= 96 * 1024; }

template <int P>
__device__ __forceinline__ void row_fold_tables(const float2* __restrict__ rlx, int V, int tid, int nt, float2* tb) {
  const int Vp = row_fold_stride(V);
  for (int i = tid; i < (P / 2 + 2) * Vp; i += nt) {
    const int k = i / Vp, l = i - k * Vp;
    tb[i] = l < V ? __ldg(rlx + (k <= P / 2 ? k * l : P * l)) : make_float2(0.f, 0.f);
  }
}

// qs: the row's bins, 16-byte aligned, zeros from nbins to the next multiple of P;
// tb: the tables above (SM) or the roots of Lx; l < V
template <int P, bool SM>
__device__ __forceinline__ void row_fold(const float2* qs, int nbins, const float2* tb, int V, int l,
                                         float2 (&Y)[P / 2 + 1]) {
  static_assert(P >= 8, "blocks of four bins or more");
  constexpr int H = P / 2, BK = H < 8 ? H : 8;
  const int Vp = row_fold_stride(V);
  auto root_u = [&](int m) { return SM ? tb[(H + 1) * Vp + m] : __ldg(tb + P * m); };
  int m = l;  // (j + 1) l mod V
  float2 un = root_u(m);
  const float4* q4 = reinterpret_cast<const float4*>(qs);
#pragma unroll
  for (int k = 0; k <= H; k += 2) {
    const float4 v = q4[k / 2];
    Y[k] = make_float2(v.x, v.y);
    if (k < H) Y[k + 1] = make_float2(v.z, v.w);
  }
  auto add = [&](float2 q, float2 u, float2& y) { y = cfma(q, u, y); };
  auto add_conj = [&](float2 q, float2 u, float2& y) {
    y.x = fmaf(q.x, u.x, fmaf(-q.y, u.y, y.x));
    y.y = fmaf(-q.x, u.y, fmaf(-q.y, u.x, y.y));
  };
#pragma unroll
  for (int b0 = H; b0 < P; b0 += BK)
    if (b0 < nbins) {
#pragma unroll
      for (int b = b0; b < b0 + BK; b += 2) {
        const float4 v = q4[b / 2];
        if (b > H) add_conj(make_float2(v.x, v.y), un, Y[P - b]);
        add_conj(make_float2(v.z, v.w), un, Y[P - b - 1]);
      }
    }
#pragma unroll 1
  for (int j0 = P; j0 < nbins; j0 += P) {
    const float2 u = un;
    m += l;
    if (m >= V) m -= V;
    un = root_u(m);
#pragma unroll
    for (int b0 = 0; b0 < P; b0 += BK)
      if (j0 + b0 < nbins) {
#pragma unroll
        for (int b = b0; b < b0 + BK; b += 2) {
          const float4 v = q4[(j0 + b) / 2];
          if (b <= H)
            add(make_float2(v.x, v.y), u, Y[b]);
          else
            add_conj(make_float2(v.x, v.y), un, Y[P - b]);
          if (b + 1 <= H)
            add(make_float2(v.z, v.w), u, Y[b + 1]);
          else
            add_conj(make_float2(v.z, v.w), un, Y[P - b - 1]);
        }
      }
  }
#pragma unroll
  for (int k = 1; k <= H; ++k) Y[k] = cmul(Y[k], SM ? tb[k * Vp + l] : __ldg(tb + k * l));
}

}  // namespace kl
