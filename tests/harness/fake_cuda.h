// A CUDA runtime of host memory for tests of host code without a GPU: the functions
// that the code under test reaches, and the number of the current device.  Symbols
// that nothing here reaches stay unresolved.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "kl_plans.h"

static int t_device = 0;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaMemcpy(void* a, const void* b, size_t n, cudaMemcpyKind) { std::memcpy(a, b, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* a, const void* b, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(a, b, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

#define CHECK(cond)                                                \
  do {                                                             \
    if (!(cond)) {                                                 \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #cond);       \
      return 1;                                                    \
    }                                                              \
  } while (0)
