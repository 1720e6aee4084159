// kl_socs_autotune tries the slice count that an untuned plan takes, so that a tuned plan
// is no slower, and reports one of 1, 2, 4 and 8: time per slice count comes from here.
#include "fake_cuda.h"

#include <algorithm>
#include <vector>

static int default_split = 1, fastest = 1;
static std::vector<int> tried;
static float elapsed = 0.f;

extern "C" {
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = elapsed; return cudaSuccess; }
}

namespace kl {
void set_error(const std::string&) {}
int spec_choose_split(const SpecGeom&, int nimg, int K) { return nimg == 6 && K >= default_split ? default_split : 1; }
size_t spec_part_elems(const SpecGeom&, int nimg, int nsplit) { return nsplit > 1 ? (size_t)nimg * nsplit : 0; }
int socs_run_forward(kl_socs_plan_s* p, const float*, int, float*, cudaStream_t, const cudaEvent_t*) {
  tried.push_back(p->tune_nsplit);
  elapsed = p->tune_nsplit == fastest ? 1.f : 2.f;
  return KL_OK;
}
}  // namespace kl

int main() {
  float buf[1];
  for (int K : {1, 5, 64})
    for (int d : {1, 3, 8, 12, 37})
      for (int f : {1, 2, 4, 8, d}) {
        if (d > K || f > K) continue;
        kl_socs_plan_s p;
        p.gen = true;
        p.K = K;
        p.nsets = 3;
        p.max_clips = 2;
        p.part_cap = 6 * 40;
        default_split = d;
        fastest = f;
        tried.clear();
        int ns = 0;
        CHECK(kl_socs_autotune(&p, buf, 2, buf, nullptr, &ns, nullptr) == KL_OK);
        CHECK(std::count(tried.begin(), tried.end(), d) > 0);
        const bool listed = f == 1 || f == 2 || f == 4 || f == 8;
        CHECK(p.tune_nsplit == f && p.tune_clips == 2);
        CHECK(listed ? ns == f : ns == 1 || ns == 2 || ns == 4 || ns == 8);
        // a plan whose sums hold the default only
        p.part_cap = kl::spec_part_elems(p.sg, 6, d);
        fastest = 0;
        CHECK(kl_socs_autotune(&p, buf, 2, buf, nullptr, &ns, nullptr) == KL_OK);
        CHECK(p.tune_nsplit == d);  // all the same: as untuned
      }
  return 0;
}
