// fft32.cuh -- a 32-point complex FFT held by one thread.
//
// The spectral stages give each thread a whole 32-point transform instead of
// spreading it over the lanes of a warp: no shuffles (a 64-point warp FFT
// spends 20 of them, at one per clock and SM), every twiddle an immediate, and
// independent butterflies to hide the FP32 latency.  32 = 4 x 8: eight 4-point
// transforms, 21 twiddles, four 8-point transforms -- about 440 FP32
// instructions for 32 outputs.
#pragma once

#include "kl_device.cuh"

namespace kl {

template <int I>
struct idx_c {
  static constexpr int value = I;
  __device__ constexpr operator int() const { return I; }
};

// f(idx_c<I>) for I in [A, B): loop indices usable as constant expressions
template <int A, int B, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (A < B) {
    f(idx_c<A>{});
    static_for<A + 1, B>(f);
  }
}

// a * e^{SIGN 2 pi i K / 32}
template <int K, int SIGN>
__device__ __forceinline__ float2 mul_w32(float2 a) {
  constexpr int k = ((K % 32) + 32) % 32;
  if constexpr (k == 0) {
    return a;
  } else if constexpr (k == 16) {
    return make_float2(-a.x, -a.y);
  } else if constexpr (k == 8 || k == 24) {
    constexpr bool plus = (k == 8) == (SIGN > 0);  // times +i or -i
    return plus ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  } else {
    constexpr float c = (float)cx::cos2pi(k, 32), s = (float)(SIGN * cx::sin2pi(k, 32));
    return make_float2(fmaf(a.x, c, -(a.y * s)), fmaf(a.x, s, a.y * c));
  }
}

template <int SIGN>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 s0 = cadd(a0, a2), d0 = csub(a0, a2), s1 = cadd(a1, a3), d1 = mul_w32<8, SIGN>(csub(a1, a3));
  a0 = cadd(s0, s1);
  a1 = cadd(d0, d1);
  a2 = csub(s0, s1);
  a3 = csub(d0, d1);
}

// 8-point transform in place, natural order in and out
template <int SIGN>
__device__ __forceinline__ void dft8(float2 (&a)[8]) {
  dft4<SIGN>(a[0], a[2], a[4], a[6]);
  dft4<SIGN>(a[1], a[3], a[5], a[7]);
  const float2 o0 = a[1], o1 = mul_w32<4, SIGN>(a[3]), o2 = mul_w32<8, SIGN>(a[5]), o3 = mul_w32<12, SIGN>(a[7]);
  const float2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6];
  a[0] = cadd(e0, o0);
  a[1] = cadd(e1, o1);
  a[2] = cadd(e2, o2);
  a[3] = cadd(e3, o3);
  a[4] = csub(e0, o0);
  a[5] = csub(e1, o1);
  a[6] = csub(e2, o2);
  a[7] = csub(e3, o3);
}

// Unnormalised 32-point DFT, sign of the exponent SIGN: input v[n] natural,
// output X[k] in v[fft32_pos(k)] (k = k1 + 4 k2 stays where 8 k1 + k2 puts it;
// the caller's unrolled indices make the permutation free).
__host__ __device__ constexpr int fft32_pos(int k) { return 8 * (k % 4) + k / 4; }

template <int SIGN>
__device__ __forceinline__ void fft32(float2 (&v)[32]) {
  // over n1 of n = n2 + 8 n1; output k1 in place of n1
  static_for<0, 8>([&](auto n2) { dft4<SIGN>(v[n2], v[n2 + 8], v[n2 + 16], v[n2 + 24]); });
  static_for<1, 4>([&](auto k1) {
    static_for<1, 8>([&](auto n2) {
      constexpr int i = 8 * decltype(k1)::value + decltype(n2)::value;
      v[i] = mul_w32<decltype(k1)::value * decltype(n2)::value, SIGN>(v[i]);
    });
  });
  static_for<0, 4>([&](auto k1) {
    constexpr int o = 8 * decltype(k1)::value;
    float2 a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = v[o + i];
    dft8<SIGN>(a);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[o + i] = a[i];
  });
}

}  // namespace kl
