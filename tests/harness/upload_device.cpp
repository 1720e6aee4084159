// kl_socs_set_kernels and _c64 of a plan on device 1 called with device 0 current: the
// scratch and the kernels that put the values in order belong on the plan's device, and
// the caller's device is current again on return.
#include "fake_cuda.h"

#include <vector>

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
size_t spec_kernel_elems(const SpecGeom& g) { return g.nbx * g.nby; }
int spec_interleave(const float* re, const float* im, size_t n, float2* H, cudaStream_t) {
  on_plan_device();
  ++launches;
  for (size_t i = 0; i < n; ++i) H[i] = make_float2(re[i], im[i]);
  return KL_OK;
}
int spec_columns(const SpecGeom& g, const float2* H, int nk, float2* HT, cudaStream_t) {
  on_plan_device();
  ++launches;
  std::memcpy(HT, H, sizeof(float2) * g.nbx * g.nby * nk);
  return KL_OK;
}
}  // namespace kl

static kl_socs_plan_s plan(int nb, int nk, float2* HT, float* lam, float2* H) {
  kl_socs_plan_s p;
  p.g.nbx = p.g.nby = p.sg.nbx = p.sg.nby = nb;
  p.K = nk;
  p.nsets = 2;
  p.device = 1;
  p.HT = HT;
  p.lam = lam;
  p.H = H;
  return p;
}

int main() {
  // sets put together on the host, at the edge of that, and above it
  for (int nb : {1, 3, 78, 79, 201})
    for (int keeps_H = 0; keeps_H < 2; ++keeps_H)
      for (int planes = 0; planes < 2; ++planes) {
        constexpr int nk = 2;
        const size_t n = (size_t)nb * nb * nk;
        std::vector<float> re(n), im(n), lam(2 * nk, -1.f);
        const float scales[nk] = {3.f, 2.f};
        std::vector<float2> both(n), HT(2 * n, make_float2(0.f, 0.f)), H(2 * n);
        for (size_t i = 0; i < n; ++i) both[i] = make_float2(re[i] = 1.f + i, im[i] = -1.f - i);
        kl_socs_plan_s p = plan(nb, nk, HT.data(), lam.data(), keeps_H ? H.data() : nullptr);
        CHECK((planes ? kl_socs_set_kernels(&p, 1, re.data(), im.data(), scales)
                      : kl_socs_set_kernels_c64(&p, 1, reinterpret_cast<float*>(both.data()), scales)) == KL_OK);
        CHECK(launches > 0);
        CHECK(wrong == 0);
        CHECK(t_device == 0);
        CHECK(held == 0);
        CHECK(std::memcmp(HT.data() + n, both.data(), sizeof(float2) * n) == 0);
        CHECK(!keeps_H || std::memcmp(H.data() + n, both.data(), sizeof(float2) * n) == 0);
        CHECK(HT[n - 1].x == 0.f && lam[0] == -1.f && lam[1] == -1.f && lam[2] == 3.f && lam[3] == 2.f);
      }
  float v[9 * 2] = {}, lam[2];
  float2 HT[9 * 2];
  kl_socs_plan_s p = plan(3, 2, HT, lam, nullptr);
  fail_alloc = true;
  CHECK(kl_socs_set_kernels(&p, 0, v, v, v) == KL_ERR_NOMEM);
  CHECK(t_device == 0 && wrong == 0);
  return 0;
}
