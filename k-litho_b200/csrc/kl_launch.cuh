// kl_launch.cuh -- programmatic dependent launch of the imaging kernels.
//
// A call is a chain of short kernels.  Each is launched so that the next one's
// CTAs may start (and set up shared memory, twiddles, kernel rings) while it still
// runs; what depends on earlier work comes after dep_wait(), which returns when
// every earlier kernel of the stream has finished and its writes are visible.
// Kernels call it before their first such access, and dep_launch() after it, so
// at most one kernel is ahead.  Of a 25 us call on one 512^2 clip the launch gaps
// are 4-5 us.
//
// A kernel that starts ahead gets the SMs its predecessor leaves free then, not an even
// share: a mask transform of one or two CTAs per SM, started at the beginning of the
// previous call's row synthesis, took twice as long.  So the general pipeline's row
// syntheses, a call's last kernels, call dep_launch() when their rows are written.
// Calls back to back, us, at the beginning and at the end: one 2004 x 1184 clip 77 / 40,
// one 2008 x 2016 64 / 39, eight 1002 x 744 81 / 58, seven 1000 x 744 at two focus values
// 94 / 86; where the transform fills the SMs the earlier start was 2 us better, eight
// 2080 x 2048 119 / 122.
//
// Such a kernel is resident while its input is still being written.  So that input is
// read by coherent loads that stay behind dep_wait(): plain ones through pointers
// without __restrict__, or __ldcs and __ldcg (volatile).  __ldg and const __restrict__
// promise data that nobody writes while the kernel runs, and such loads may be moved
// above the wait; they are for the plan's tables and kernels only.
#pragma once

#include <cuda_runtime.h>

#include "kl_early.h"

namespace kl {

__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = t_early_launch ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace kl
