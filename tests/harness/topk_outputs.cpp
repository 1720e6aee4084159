// Top-K solves that fail after their host work was done: the caller's arrays are as they
// were; and a solve that succeeds touches no byte beyond them.
#include "fake_cuda.h"

#include <vector>

static int rc_solve = KL_ERR_NOT_CONVERGED, calls = 0;

namespace kl {
void set_error(const std::string&) {}
int scratch_alloc(void** p, size_t bytes, cudaStream_t, const char*) {
  *p = std::calloc(1, bytes);
  return KL_OK;
}
void scratch_free(void* p, cudaStream_t) { std::free(p); }
int eig_topk_factor(const float2*, int, int, const EigenOptions&, double2*, double*, EigenResult*, cudaStream_t,
                    const std::function<void()>& meanwhile) {
  ++calls;
  if (meanwhile) meanwhile();
  return rc_solve;
}
int eig_topk_factor_batch(const std::vector<FactorProblem>&, const EigenOptions&, cudaStream_t,
                          const std::function<void()>& meanwhile) {
  ++calls;
  if (meanwhile) meanwhile();
  return rc_solve;
}
int eig_to_kernels(const double2*, int N, int K, float* re, float* im, cudaStream_t) {
  for (int i = 0; i < N * K * (im ? 1 : 2); ++i) re[i] = 7.f;
  for (int i = 0; im && i < N * K; ++i) im[i] = 8.f;
  return KL_OK;
}
}  // namespace kl

int main() {
  constexpr int N = 5000, nk = 3, guard = 4096;
  kl_tcc_plan_s a, b;
  for (kl_tcc_plan_s* p : {&a, &b}) {
    p->pp.N = N;
    p->pp.S = 100;
  }
  const kl_tcc_plan plans[2] = {&a, &b};
  for (int batch = 0; batch < 2; ++batch)
    for (int c64 = 0; c64 < 2; ++c64) {
      const size_t n = (size_t)N * nk * (batch ? 2 : 1);
      std::vector<float> re(n * (c64 ? 2 : 1) + guard, 1.5f), im(n + guard, -2.5f), scales(2 * nk, 3.f);
      std::vector<double> ev(2 * nk, 4.0);
      int it[2] = {-1, -1};
      const std::vector<float> re0 = re, im0 = im, sc0 = scales;
      auto solve = [&] {
        if (batch)
          return c64 ? kl_topk_eig_batch_c64(plans, 2, nk, 0, re.data(), scales.data(), ev.data(), it)
                     : kl_topk_eig_batch(plans, 2, nk, 0, re.data(), im.data(), scales.data(), ev.data(), it);
        return c64 ? kl_topk_eig_c64(&a, nk, 0, re.data(), scales.data(), ev.data(), it)
                   : kl_topk_eig(&a, nk, 0, re.data(), im.data(), scales.data(), ev.data(), it);
      };
      rc_solve = KL_ERR_NOT_CONVERGED;
      calls = 0;
      CHECK(solve() == KL_ERR_NOT_CONVERGED);
      CHECK(calls == 1);
      CHECK(re == re0);
      CHECK(im == im0);
      CHECK(scales == sc0 && ev[0] == 4.0 && it[0] == -1);
      rc_solve = KL_OK;
      CHECK(solve() == KL_OK);
      for (size_t i = 0; i < re.size(); ++i) CHECK(re[i] == (i + guard < re.size() ? 7.f : 1.5f));
      for (size_t i = 0; i < im.size(); ++i) CHECK(im[i] == (!c64 && i + guard < im.size() ? 8.f : -2.5f));
    }
  return 0;
}
