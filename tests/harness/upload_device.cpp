// kl_socs_set_kernels and _c64 of a plan on device 1 called with device 0 current: the
// scratch and the kernels that put the values in order belong on the plan's device, and
// the caller's device is current again on return.
#include "fake_cuda.h"

static int wrong = 0, launches = 0, allocs = 0, held = 0;
static bool fail_alloc = false;
static void on_plan_device() { wrong += t_device != 1; }

namespace kl {
void set_error(const std::string&) {}
int scratch_alloc(void** p, size_t bytes, cudaStream_t, const char*) {
  on_plan_device();
  ++allocs;
  if (fail_alloc) return KL_ERR_NOMEM;
  *p = std::malloc(bytes);
  ++held;
  return KL_OK;
}
void scratch_free(void* p, cudaStream_t) {
  on_plan_device();
  std::free(p);
  --held;
}
size_t spec_kernel_elems(const SpecGeom&) { return 9; }
int spec_interleave(const float* re, const float* im, size_t n, float2* H, cudaStream_t) {
  on_plan_device();
  ++launches;
  for (size_t i = 0; i < n; ++i) H[i] = make_float2(re[i], im[i]);
  return KL_OK;
}
int spec_columns(const SpecGeom&, const float2* H, int nk, float2* HT, cudaStream_t) {
  on_plan_device();
  ++launches;
  std::memcpy(HT, H, sizeof(float2) * 9 * nk);
  return KL_OK;
}
}  // namespace kl

int main() {
  constexpr int n = 9, nk = 2;
  float re[n * nk], im[n * nk], scales[nk] = {3.f, 2.f}, lam[nk];
  float2 both[n * nk], HT[n * nk], H[n * nk];
  for (int i = 0; i < n * nk; ++i) both[i] = make_float2(re[i] = 1.f + i, im[i] = -1.f - i);
  for (int keeps_H = 0; keeps_H < 2; ++keeps_H)
    for (int planes = 0; planes < 2; ++planes) {
      kl_socs_plan_s p;
      p.g.nbx = p.g.nby = 3;
      p.K = nk;
      p.nsets = 1;
      p.device = 1;
      p.HT = HT;
      p.lam = lam;
      p.H = keeps_H ? H : nullptr;
      std::memset(HT, 0, sizeof(HT));
      const int l0 = launches;
      CHECK((planes ? kl_socs_set_kernels(&p, 0, re, im, scales)
                    : kl_socs_set_kernels_c64(&p, 0, reinterpret_cast<float*>(both), scales)) == KL_OK);
      CHECK(launches - l0 == 1 + planes);
      CHECK(wrong == 0);
      CHECK(t_device == 0);
      CHECK(held == 0);
      CHECK(std::memcmp(HT, both, sizeof(both)) == 0);
      CHECK(lam[0] == 3.f && lam[1] == 2.f);
    }
  kl_socs_plan_s p;
  p.g.nbx = p.g.nby = 3;
  p.K = nk;
  p.nsets = 1;
  p.device = 1;
  p.HT = HT;
  p.lam = lam;
  fail_alloc = true;
  CHECK(kl_socs_set_kernels(&p, 0, re, im, scales) == KL_ERR_NOMEM);
  CHECK(t_device == 0 && wrong == 0);
  return 0;
}
