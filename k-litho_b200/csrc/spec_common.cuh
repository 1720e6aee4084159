// spec_common.cuh -- pieces shared by the spectral cores of the image (spectral.cuh)
// and of the adjoint (adjoint_spectral.cu): roots of unity, the layout of the
// kernels and their cp.async feed.
#pragma once

#include "fft32.cuh"
#include "kl_internal.h"
#include "kl_launch.cuh"

namespace kl {
namespace spec {

constexpr int kP = 33;  // pitch of 32-wide rows

// e^{+2 pi i m / G}
template <int G>
struct RootTable {
  float c[G], s[G];
  constexpr RootTable() : c(), s() {
    for (int k = 0; k < G; ++k) {
      c[k] = (float)cx::cos2pi(k, G);
      s[k] = (float)cx::sin2pi(k, G);
    }
  }
};
template <int G>
__device__ const RootTable<G> g_roots = RootTable<G>();

// one kernel in the core's layout: n = 0 for every row (padded to 16 bytes), then
// [group][sign][pair][row][2]
__host__ __device__ inline int spec_n0(const SpecGeom& g) { return g.nby + 1; }
__host__ __device__ inline size_t spec_hstride(const SpecGeom& g) {
  return (size_t)spec_n0(g) + (size_t)(g.G / 16) * 8 * g.nby;
}

__device__ __forceinline__ void cp_async16(unsigned dst, const float2* src, int bytes) {
  // bytes = 0: the slot is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// The kernel values of one row thread, group by group, for the thread's kernel
// of every batch.
template <int RING, int NQ, int ROW>
struct RowFeed {
  const float2* h;      // the next group of the thread's row
  ptrdiff_t pair, skip; // strides of a pair, and from the last group of a kernel to the next batch's first
  unsigned ring;        // shared address of this thread's slot 0
  int q, put;
  int left, bytes;      // batches for which the thread's slot holds a kernel; 16, or 0 after them
  __device__ __forceinline__ void push() {
    const unsigned d = ring + put * (8 * ROW * 8);
#pragma unroll
    for (int i = 0; i < 4; ++i) cp_async16(d + i * (2 * ROW * 8), h + i * pair, bytes);
    cp_commit();
    put = put + 1 == RING ? 0 : put + 1;
    if (++q == NQ) {
      q = 0;
      if (--left > 0) h += 4 * pair + skip;
      else bytes = 0;
    } else if (bytes) {
      h += 4 * pair;
    }
  }
};

template <int G>
__device__ __forceinline__ float2 root_of(int m) {
  int q = m % G;
  q = q < 0 ? q + G : q;
  return make_float2(g_roots<G>.c[q], g_roots<G>.s[q]);
}

}  // namespace spec
}  // namespace kl
