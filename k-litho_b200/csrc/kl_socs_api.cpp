// kl_socs_api.cpp -- C ABI for SOCS imaging plans (see include/klitho_gpu.h).
#include <cuda_runtime.h>

#include <cstdint>
#include <algorithm>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "kl_internal.h"
#include "kl_early.h"
#include "kl_plans.h"

namespace {
void drop_events(kl_socs_plan p) {
  for (cudaEvent_t e : p->events) cudaEventDestroy(e);
  p->events.clear();
}

void free_plan(kl_socs_plan p) {
  if (!p) return;
  drop_events(p);
  for (int i = 0; i < 3; ++i) {
    if (p->hs[i]) {
      cudaStreamSynchronize(p->hs[i]);
      cudaStreamDestroy(p->hs[i]);
    }
    if (p->hev[i]) cudaEventDestroy(p->hev[i]);
  }
  cudaFree(p->buffers);
  cudaFree(p->stage_in);
  cudaFree(p->stage_out);
  delete p;
}

// A plan's device buffers are pieces of one allocation: every cudaMalloc costs
// 0.1 ms and more, and a plan made inside a call (kl_hopkins_image) pays for it.
struct Pieces {
  std::vector<std::pair<void**, size_t>> list;
  template <typename T>
  void add(T** p, size_t bytes) {
    list.emplace_back(reinterpret_cast<void**>(p), (std::max<size_t>(bytes, 16) + 255) & ~size_t(255));
  }
  int allocate(void** base) const;
};

int alloc(void** ptr, size_t bytes, const char* what) {
  cudaError_t e = cudaMalloc(ptr, bytes ? bytes : 16);
  if (e != cudaSuccess) {
    kl::set_error(std::string("cudaMalloc(") + what + "): " + cudaGetErrorString(e));
    cudaGetLastError();
    return KL_ERR_NOMEM;
  }
  return KL_OK;
}

int Pieces::allocate(void** base) const {
  size_t total = 0;
  for (const auto& e : list) total += e.second;
  if (int rc = alloc(base, total, "plan buffers")) return rc;
  char* c = static_cast<char*>(*base);
  for (const auto& e : list) {
    *e.first = c;
    c += e.second;
  }
  return KL_OK;
}

int mark(kl_socs_plan p, cudaStream_t st) {
  if (!p->timing) return KL_OK;
  cudaEvent_t e;
  KL_CUDA_TRY(cudaEventCreate(&e));
  p->events.push_back(e);
  KL_CUDA_TRY(cudaEventRecord(e, st));
  return KL_OK;
}

int stage_mark(kl_socs_plan p, cudaStream_t st, const cudaEvent_t* ev4, int i) {
  if (!ev4) return mark(p, st);
  // inside a stream capture the record must become an event node of the graph
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  KL_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
  KL_CUDA_TRY(cudaEventRecordWithFlags(ev4[i], st,
                                       cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal
                                                                           : cudaEventRecordDefault));
  return KL_OK;
}

// the launch shape for a batch of nclips: the autotuned one when it was tuned
// for this batch size, else the heuristic
void launch_shape(kl_socs_plan p, int nclips, int* nsplit, int* spc) {
  if (p->tune_clips == nclips && p->tune_nsplit > 0) {
    *nsplit = p->tune_nsplit;
    *spc = p->tune_spc;
  } else {
    *nsplit = kl::spec_choose_split(p->sg, nclips * p->nsets, p->K);
    *spc = 0;
  }
}

// general-geometry pipeline: row transform, column transform, spectral core,
// column synthesis, row synthesis
int run_forward_gen(kl_socs_plan p, const float* masks, int nclips, float* images, cudaStream_t st,
                    const cudaEvent_t* ev4) {
  const kl::GenGeom& g = p->gg;
  const int nimg = nclips * p->nsets;
  int nsplit, spc;
  launch_shape(p, nclips, &nsplit, &spc);
  const int nparts = kl::gen_choose_parts(g, nclips, g.nf);
  int rc;
  if ((rc = stage_mark(p, st, ev4, 0))) return rc;
  if ((rc = kl::gen_launch_rowfwd(g, p->gtab, masks, nclips * g.Ly, p->R, st))) return rc;
  if ((rc = kl::gen_launch_colfwd(g, p->gtab, p->R, nclips, g.nf, g.Ny, 1.0f / ((float)g.Lx * (float)g.Ly), nparts,
                                  p->band, st)))
    return rc;
  if ((rc = stage_mark(p, st, ev4, 1))) return rc;
  if ((rc = kl::spec_launch(p->sg, p->band, nparts, 1.0f, nimg, p->HT, false, p->lam, p->K, p->nsets, nsplit, p->part,
                            p->T, p->done, st)))
    return rc;
  if ((rc = stage_mark(p, st, ev4, 2))) return rc;
  if ((rc = kl::gen_launch_colinv(g, p->gtab, p->T, nimg, 2 * g.Ny, g.ntx, p->Q, st))) return rc;
  if ((rc = kl::gen_launch_rowinv(g, p->gtab, p->Q, nimg, g.ntx, images, st))) return rc;
  return stage_mark(p, st, ev4, 3);
}

// synthesis on the tensor cores for a batch of nclips clips: when requested,
// or when the autotuner picked it for this batch size
bool use_tc_synthesis(kl_socs_plan p, int nclips) {
  if (p->gen || !p->bhi) return false;
  if (p->synth == KL_SYNTH_TENSOR_CORES) return true;
  if (p->synth == KL_SYNTH_CUDA_CORES) return false;
  return p->tune_clips == nclips && p->tune_nsplit > 0 && p->tune_spc < 0;
}

// mask transform on the tensor cores: with the tensor-core engine forced, or
// when the autotuner picked it (tune_spc == -2) for this batch size
bool use_tc_forward(kl_socs_plan p, int nclips, const float* masks) {
  if (p->gen || !p->thi || !kl::fwd_tc_supported(p->g) || ((uintptr_t)masks & 15)) return false;
  if (p->synth == KL_SYNTH_TENSOR_CORES) return true;
  if (p->synth == KL_SYNTH_CUDA_CORES) return false;
  return p->tune_clips == nclips && p->tune_nsplit > 0 && p->tune_spc == -2;
}

// the spectral core of the specialised pipeline, from the strip partials
int spectral(kl_socs_plan p, int nclips, int nsplit, cudaStream_t st) {
  return kl::spec_launch(p->sg, p->partial, p->g.nS, 1.0f / ((float)p->g.Lx * (float)p->g.Ly), nclips * p->nsets, p->HT,
                         false, p->lam, p->K, p->nsets, nsplit, p->part, p->T, p->done, st);
}

// buffers of the spectral core: the kernels in its layout (and, for the adjoint on
// grids above 128 points, the kernel layout), spectra for any batch up to max_clips, slice counters
void spectral_pieces(kl_socs_plan p, Pieces& mem) {
  const kl::SpecGeom& g = p->sg;
  const size_t nk = (size_t)p->K * p->nsets, nimg = (size_t)p->max_clips * p->nsets;
  for (int n = 1; n <= p->max_clips; ++n)
    p->part_cap = std::max(p->part_cap, kl::spec_part_elems(g, n * p->nsets,
                                                            kl::spec_choose_split(g, n * p->nsets, p->K)));
  mem.add(&p->HT, sizeof(float2) * nk * kl::spec_kernel_elems(g));
  if (p->adjoint && !kl::adjoint_core(g)) mem.add(&p->H, sizeof(float2) * nk * g.nby * g.nbx);
  mem.add(&p->lam, sizeof(float) * nk);
  mem.add(&p->T, sizeof(float2) * nimg * g.nty * g.ntx);
  mem.add(&p->part, sizeof(float2) * p->part_cap);
  mem.add(&p->done, sizeof(unsigned) * nimg);
}

// kernel slices of the adjoint's spectral stage, and its shares of Gam per image
int adjoint_split(kl_socs_plan p, int nimg) {
  return kl::adjoint_core(p->sg) ? kl::adjoint_choose_split(p->sg, nimg, p->K) : kl::gen_choose_split(p->gg, nimg, p->K);
}
int adjoint_parts(kl_socs_plan p, int nsplit) {
  return kl::adjoint_core(p->sg) ? nsplit * kl::adjoint_shares(p->sg) : nsplit;
}
// the largest number of shares any batch size needs
size_t adjoint_shares_cap(kl_socs_plan p) {
  size_t cap = 0;
  for (int n = 1; n <= p->max_clips; ++n) {
    const int nimg = n * p->nsets;
    cap = std::max(cap, (size_t)nimg * adjoint_parts(p, adjoint_split(p, nimg)));
  }
  return cap;
}

// a new plan's kernels are zero, as are its counters; the default stream's work
// is done on return
int finish_plan(kl_socs_plan p) {
  const kl::SpecGeom& g = p->sg;
  const size_t nk = (size_t)p->K * p->nsets;
  cudaMemsetAsync(p->HT, 0, sizeof(float2) * nk * kl::spec_kernel_elems(g), nullptr);
  if (p->H) cudaMemsetAsync(p->H, 0, sizeof(float2) * nk * g.nby * g.nbx, nullptr);
  cudaMemsetAsync(p->lam, 0, sizeof(float) * nk, nullptr);
  cudaMemsetAsync(p->done, 0, sizeof(unsigned) * p->max_clips * p->nsets, nullptr);
  if (p->status) cudaMemsetAsync(p->status, 0, sizeof(int), nullptr);
  if (cudaStreamSynchronize(nullptr) != cudaSuccess) {
    kl::set_error(std::string("kl_socs_plan_create: ") + cudaGetErrorString(cudaGetLastError()));
    return KL_ERR_CUDA;
  }
  return KL_OK;
}

int run_forward(kl_socs_plan p, const float* masks, int nclips, float* images, cudaStream_t st,
                const cudaEvent_t* ev4 = nullptr) {
  const kl::EarlyLaunch early(!ev4 && !p->timing);
  if (p->gen) return run_forward_gen(p, masks, nclips, images, st, ev4);
  int rc;
  if ((rc = stage_mark(p, st, ev4, 0))) return rc;
  int nsplit, spc;
  launch_shape(p, nclips, &nsplit, &spc);
  const bool tc = use_tc_synthesis(p, nclips) && kl::synth_tc_aligned(images);
  spc = spc > 0 ? spc : 0;
  if (use_tc_forward(p, nclips, masks))
    rc = kl::fwd_tc_launch(p->g, masks, nclips, p->ty, p->thi, p->tlo, p->partial, p->status, st);
  else
    rc = kl::socs_launch_forward(p->g, p->tx, p->ty, masks, nclips, p->partial, st);
  if (rc) return rc;
  if ((rc = stage_mark(p, st, ev4, 1))) return rc;
  rc = spectral(p, nclips, nsplit, st);
  if (rc) return rc;
  if ((rc = stage_mark(p, st, ev4, 2))) return rc;
  rc = tc ? kl::synth_tc_launch(p->g, p->T, p->ty, p->bhi, p->blo, nclips * p->nsets, images, p->status, st)
          : kl::socs_launch_inverse(p->g, p->tx, p->ty, p->T, nclips, p->nsets, images, st, spc);
  if (rc) return rc;
  return stage_mark(p, st, ev4, 3);
}
// plan on the general-geometry pipeline
int create_gen_plan(kl_socs_plan* plan, int Lx, int Ly, int Nx, int Ny, int nk, int nsets, int max_clips,
                    bool adjoint) {
  kl::GenGeom gg;
  int rc = kl::gen_geometry(Lx, Ly, Nx, Ny, &gg);
  if (rc) return rc;
  kl_socs_plan p = new (std::nothrow) kl_socs_plan_s;
  if (!p) {
    kl::set_error("kl_socs_plan_create: out of host memory");
    return KL_ERR_NOMEM;
  }
  p->gen = true;
  p->adjoint = adjoint;
  p->gg = gg;
  // sizes only, for callers that read them
  p->g.Lx = Lx;
  p->g.Ly = Ly;
  p->g.Nx = Nx;
  p->g.Ny = Ny;
  p->g.nbx = gg.nbx;
  p->g.nby = gg.nby;
  p->g.nf = gg.nf;
  p->g.ntx = gg.ntx;
  p->g.nty = gg.nty;
  p->g.G = gg.G;
  p->g.nS = gg.nS;
  p->g.dx = gg.dx;
  p->g.dy = gg.dy;
  p->K = nk;
  p->nsets = nsets;
  p->max_clips = max_clips;
  cudaGetDevice(&p->device);
  p->sg = kl::spec_geometry(gg);
  int pmax = 0;
  for (int n = 1; n <= max_clips; ++n) pmax = std::max(pmax, kl::gen_choose_parts(gg, n, gg.nf));
  p->nparts_max = pmax;
  Pieces mem;
  spectral_pieces(p, mem);
  mem.add(&p->gtab, sizeof(float2) * kl::gen_table_elems(gg));
  mem.add(&p->R, kl::gen_rowbins_bytes(gg, max_clips, gg.nf));
  mem.add(&p->band, kl::gen_band_bytes(gg, max_clips, pmax, gg.nby, gg.nf));
  mem.add(&p->Q, kl::gen_rowbins_bytes(gg, max_clips * nsets, gg.ntx));
  if (adjoint) {
    int gmax = 0;
    for (int n = 1; n <= max_clips; ++n) gmax = std::max(gmax, kl::gen_choose_parts(gg, n * nsets, gg.ntx));
    p->gparts_max = gmax;
    mem.add(&p->gband, kl::gen_band_bytes(gg, max_clips * nsets, gmax, gg.nty, gg.ntx));
    mem.add(&p->gamma, sizeof(float) * kl::adjoint_gamma_elems(p->sg, max_clips * nsets));
    mem.add(&p->gam, sizeof(float2) * gg.nby * gg.nbx * adjoint_shares_cap(p));
    mem.add(&p->Tg, sizeof(float2) * (size_t)max_clips * gg.nf * gg.nby);
  }
  if ((rc = mem.allocate(&p->buffers)) || (rc = kl::gen_build_tables(gg, p->gtab, nullptr)) || (rc = finish_plan(p))) {
    free_plan(p);
    return rc;
  }
  *plan = p;
  return KL_OK;
}

int create_plan(kl_socs_plan* plan, int Lx, int Ly, int Nx, int Ny, int nk, int nsets,
                int max_clips, bool adjoint, bool general = false) {
  KL_CHECK_ARG(plan != nullptr, "kl_socs_plan_create: plan is NULL");
  *plan = nullptr;
  KL_CHECK_ARG(nk > 0 && nsets > 0 && max_clips > 0, "kl_socs_plan_create: nk, nsets, max_clips must be positive");
  kl::SocsGeom g;
  int rc = general ? KL_ERR_UNSUPPORTED : kl::socs_geometry(Lx, Ly, Nx, Ny, &g, adjoint);
  if (!rc && adjoint) rc = kl::vjp_supported(g);
  // geometries outside the specialised kernels run on the general pipeline
  if (rc == KL_ERR_UNSUPPORTED) return create_gen_plan(plan, Lx, Ly, Nx, Ny, nk, nsets, max_clips, adjoint);
  if (rc) return rc;
  kl_socs_plan p = new (std::nothrow) kl_socs_plan_s;
  if (p) p->adjoint = adjoint;
  if (!p) {
    kl::set_error("kl_socs_plan_create: out of host memory");
    return KL_ERR_NOMEM;
  }
  p->g = g;
  p->K = nk;
  p->nsets = nsets;
  p->max_clips = max_clips;
  cudaGetDevice(&p->device);
  p->sg = kl::spec_geometry(g);
  Pieces mem;
  spectral_pieces(p, mem);
  mem.add(&p->partial, kl::socs_partial_bytes(g, max_clips));
  mem.add(&p->tx, sizeof(float2) * kl::socs_table_x_elems(g));
  mem.add(&p->ty, sizeof(float2) * kl::socs_table_y_elems(g));
  if (kl::synth_tc_supported(g)) {
    const size_t bb = (size_t)g.Lx * kl::synth_tc_kp(g) * 2;
    mem.add(&p->bhi, bb);
    mem.add(&p->blo, bb);
    mem.add(&p->status, sizeof(int));
    // the transposed basis of the row DFTs: the tensor-core mask transform and,
    // on adjoint plans, the row DFT of dL/dI
    p->vjp_tc = adjoint && kl::synth_tc_kp(g) == 64 && kl::vjp_tc_supported(g);
    if (kl::fwd_tc_supported(g) || p->vjp_tc) {
      const size_t tb = (size_t)64 * g.Lx * 2;
      mem.add(&p->thi, tb);
      mem.add(&p->tlo, tb);
    }
  }
  if (adjoint) {
    mem.add(&p->gpart, kl::vjp_gpart_bytes(g, max_clips * nsets));
    mem.add(&p->gamma, sizeof(float) * kl::adjoint_gamma_elems(p->sg, max_clips * nsets));
    mem.add(&p->gam, sizeof(float2) * g.nby * g.nbx * adjoint_shares_cap(p));
    mem.add(&p->Tg, sizeof(float2) * (size_t)max_clips * g.nty * g.ntx);
  }
  if ((rc = mem.allocate(&p->buffers)) || (rc = kl::socs_build_tables(g, p->tx, p->ty, nullptr)) ||
      (p->bhi && (rc = kl::synth_tc_build_basis(g, p->bhi, p->blo, nullptr))) ||
      (p->thi && (rc = kl::vjp_tc_build_basis_t(g, p->thi, p->tlo, nullptr))) || (rc = finish_plan(p))) {
    free_plan(p);
    return rc;
  }
  *plan = p;
  return KL_OK;
}
}  // namespace

namespace {
// adjoint on the general pipeline: forward to T, image + resist + dL/dI row
// bins, dL/dI band, Gam, gradient spectrum, gradient image
int vjp_gen(kl_socs_plan p, const float* masks, const float* targets, int nclips, float alpha, float threshold,
            float* images, float* grad, double* loss, cudaStream_t st) {
  const kl::GenGeom& g = p->gg;
  const int nimg = nclips * p->nsets;
  const int ns = kl::spec_choose_split(p->sg, nimg, p->K);
  const int ns_adj = adjoint_split(p, nimg);
  const int nparts = kl::gen_choose_parts(g, nclips, g.nf);
  const int gparts = kl::gen_choose_parts(g, nimg, g.ntx);
  int rc;
  if ((rc = kl::gen_launch_rowfwd(g, p->gtab, masks, nclips * g.Ly, p->R, st))) return rc;
  if ((rc = kl::gen_launch_colfwd(g, p->gtab, p->R, nclips, g.nf, g.Ny, 1.0f / ((float)g.Lx * (float)g.Ly), nparts,
                                  p->band, st)))
    return rc;
  if ((rc = kl::spec_launch(p->sg, p->band, nparts, 1.0f, nimg, p->HT, false, p->lam, p->K, p->nsets, ns, p->part, p->T,
                            p->done, st)))
    return rc;
  if ((rc = kl::gen_launch_colinv(g, p->gtab, p->T, nimg, 2 * g.Ny, g.ntx, p->Q, st))) return rc;
  KL_CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(double) * (size_t)nimg, st));
  // image, then dL/dI's row bins from it; without a place for the image (no output
  // for it, several images per clip, an output over the targets, which are still to be
  // read) both in one kernel.  The gradient is written last
  float* im = images ? images : p->nsets == 1 ? grad : nullptr;
  const size_t px = (size_t)g.Lx * g.Ly;
  const bool over = im && im < targets + px * nclips && targets < im + px * nimg;
  if (kl::gen_direct_dft(g) && im && !over) {
    const float2* rlx = kl::gen_roots_x(g, p->gtab);
    if ((rc = kl::row_synth(g, rlx, p->Q, nimg * g.Ly, g.ntx, im, st))) return rc;
    rc = kl::row_dft_vjp(g, rlx, im, nimg, g.ntx, targets, p->nsets, alpha, threshold, loss, p->Q, st);
  } else {
    rc = kl::gen_launch_rowvjp(g, p->gtab, p->Q, nimg, p->nsets, targets, alpha, threshold, images, loss, st);
  }
  if (rc) return rc;
  if ((rc = kl::gen_launch_colfwd(g, p->gtab, p->Q, nimg, g.ntx, 2 * g.Ny, 1.0f, gparts, p->gband, st))) return rc;
  rc = kl::adjoint_core(p->sg)
           ? kl::adjoint_launch(p->sg, p->band, nparts, 1.0f, p->gband, gparts, nimg, p->HT, p->lam, p->K, p->nsets, ns_adj,
                                p->gamma, p->gam, st)
           : kl::gen_launch_vjp_spectral(g, p->band, nparts, p->gband, gparts, nclips, p->H, p->lam, p->K, p->nsets,
                                         ns_adj, p->gam, st);
  if (rc) return rc;
  if ((rc = kl::adjoint_gradient(p->sg, p->gam, nclips, p->nsets * adjoint_parts(p, ns_adj), g.Ny, g.nf, 1, g.nby, p->Tg,
                                 st)))
    return rc;
  if ((rc = kl::gen_launch_colinv(g, p->gtab, p->Tg, nclips, g.Ny, g.nf, p->Q, st))) return rc;
  if ((rc = kl::gen_launch_rowinv(g, p->gtab, p->Q, nclips, g.nf, grad, st))) return rc;
  p->last_vjp_clips = nclips;
  p->last_nparts = nparts;
  p->last_gparts = gparts;
  return KL_OK;
}
}  // namespace

namespace {
// kernels of one set from the host, interleaved (im null) or as two planes: copied as
// they are and put in order on the device -- interleaving 6 MB on the host took
// longer than the copy.  Sets up to kPackElems are put together with their eigenvalues on
// the host instead: a copy from pageable memory takes about 10 us whatever its size (two
// planes of 2312, 6936 and 12696 values: 37, 42 and 46 us by three copies, 25, 34 and 47
// put together).
// The kernel layout is kept where an adjoint needs it, else only on the way to the
// spectral core's.  On the plan's device, whichever is current.  Done on return.
constexpr size_t kPackElems = 12288;
int upload_kernels(kl_socs_plan p, int set, const float* re, const float* im, const float* scales) {
  const kl::OnDevice on(p->device);
  KL_CUDA_TRY(on.status);
  const size_t n = (size_t)p->g.nby * p->g.nbx * p->K, k0 = (size_t)set * p->K;
  const bool pack = n <= kPackElems && !p->H;
  void* tmp = nullptr;
  const size_t tmp_floats = pack ? 2 * n + p->K : (p->H ? 0 : 2 * n) + (im ? 2 * n : 0);
  int rc = tmp_floats ? kl::scratch_alloc(&tmp, sizeof(float) * tmp_floats, nullptr, "kernels") : KL_OK;
  if (rc) return rc;
  float2* H = p->H ? p->H + set * n : static_cast<float2*>(tmp);
  float* planes = static_cast<float*>(tmp) + (p->H ? 0 : 2 * n);
  auto copy = [&](void* dst, const void* src, size_t bytes, cudaMemcpyKind kind = cudaMemcpyHostToDevice) {
    const cudaError_t e = kind == cudaMemcpyHostToDevice ? cudaMemcpy(dst, src, bytes, kind)
                                                         : cudaMemcpyAsync(dst, src, bytes, kind, nullptr);
    if (e == cudaSuccess) return KL_OK;
    kl::set_error(std::string("kl_socs_set_kernels: ") + cudaGetErrorString(e));
    return KL_ERR_CUDA;
  };
  if (pack) {
    std::vector<float> h(tmp_floats);
    if (im) {
      for (size_t i = 0; i < n; ++i) {
        h[2 * i] = re[i];
        h[2 * i + 1] = im[i];
      }
    } else {
      std::memcpy(h.data(), re, sizeof(float2) * n);
    }
    std::memcpy(h.data() + 2 * n, scales, sizeof(float) * p->K);
    rc = copy(tmp, h.data(), sizeof(float) * tmp_floats);
  } else if (im) {
    if (!(rc = copy(planes, re, sizeof(float) * n)) && !(rc = copy(planes + n, im, sizeof(float) * n)))
      rc = kl::spec_interleave(planes, planes + n, n, H, nullptr);
  } else {
    rc = copy(H, re, sizeof(float2) * n);
  }
  if (!rc) rc = kl::spec_columns(p->sg, H, p->K, p->HT + k0 * kl::spec_kernel_elems(p->sg), nullptr);
  if (!rc)
    rc = pack ? copy(p->lam + k0, H + n, sizeof(float) * p->K, cudaMemcpyDeviceToDevice)
              : copy(p->lam + k0, scales, sizeof(float) * p->K);
  if (!rc && cudaStreamSynchronize(nullptr) != cudaSuccess) {
    kl::set_error(std::string("kl_socs_set_kernels: ") + cudaGetErrorString(cudaGetLastError()));
    rc = KL_ERR_CUDA;
  }
  if (tmp) kl::scratch_free(tmp, nullptr);
  return rc;
}
}  // namespace

int kl::socs_run_forward(kl_socs_plan_s* p, const float* masks, int nclips, float* images, cudaStream_t st,
                         const cudaEvent_t* ev4) {
  return run_forward(p, masks, nclips, images, st, ev4);
}

extern "C" {

int kl_socs_plan_create(kl_socs_plan* plan, int Lx, int Ly, int Nx, int Ny, int nk, int nsets,
                        int max_clips) {
  return create_plan(plan, Lx, Ly, Nx, Ny, nk, nsets, max_clips, false);
}

int kl_socs_plan_create_adjoint(kl_socs_plan* plan, int Lx, int Ly, int Nx, int Ny, int nk,
                                int nsets, int max_clips) {
  return create_plan(plan, Lx, Ly, Nx, Ny, nk, nsets, max_clips, true);
}

int kl_socs_plan_create_ex(kl_socs_plan* plan, int Lx, int Ly, int Nx, int Ny, int nk, int nsets,
                           int max_clips, int flags) {
  KL_CHECK_ARG((flags & ~(KL_SOCS_ADJOINT | KL_SOCS_GENERAL)) == 0, "kl_socs_plan_create_ex: unknown flags");
  return create_plan(plan, Lx, Ly, Nx, Ny, nk, nsets, max_clips, (flags & KL_SOCS_ADJOINT) != 0,
                     (flags & KL_SOCS_GENERAL) != 0);
}

int kl_socs_plan_engine(kl_socs_plan plan) { return plan ? (plan->gen ? 1 : 0) : -1; }

int kl_socs_vjp(kl_socs_plan p, const float* masks, const float* targets, int nclips, float alpha,
                float threshold, float* images, float* grad, double* loss, void* stream) {
  KL_CHECK_ARG(p && masks && targets && grad && loss, "kl_socs_vjp: NULL argument");
  KL_CHECK_ARG((reinterpret_cast<uintptr_t>(targets) & 15) == 0, "kl_socs_vjp: targets_dev must be 16-byte aligned");
  KL_CHECK_ARG(p->adjoint, "kl_socs_vjp: the plan was not created by kl_socs_plan_create_adjoint");
  KL_CHECK_ARG(nclips >= 0 && nclips <= p->max_clips, "kl_socs_vjp: nclips exceeds the plan");
  cudaStream_t st = (cudaStream_t)stream;
  if (nclips == 0) return KL_OK;
  if (p->gen) return vjp_gen(p, masks, targets, nclips, alpha, threshold, images, grad, loss, st);
  const kl::SocsGeom& g = p->g;
  int rc;
  if (p->synth == KL_SYNTH_TENSOR_CORES && use_tc_forward(p, nclips, masks))
    rc = kl::fwd_tc_launch(g, masks, nclips, p->ty, p->thi, p->tlo, p->partial, p->status, st);
  else
    rc = kl::socs_launch_forward(g, p->tx, p->ty, masks, nclips, p->partial, st);
  if (rc) return rc;
  if ((rc = spectral(p, nclips, kl::spec_choose_split(p->sg, nclips * p->nsets, p->K), st))) return rc;
  KL_CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(double) * (size_t)nclips * p->nsets, st));
  // image, resist, loss and the row DFT of dL/dI, and the gradient's synthesis: on the
  // tensor cores where the plan has them, unless it asks for the CUDA-core engine.  Their
  // kernels have a CTA per one or two tiles of 128 rows, the CUDA cores' one per 32 rows:
  // up to 64 image tiles those are faster, us a call of 1, 8, 12 and 32 clips (tensor
  // cores first): 512^2 99 / 74, 96 / 74, 100 / 86 (48 tiles), 107 / 117; 1024^2 160 / 131,
  // 163 / 137 (64 tiles), 172 / 166, 254 / 260; 768^2 141 / 141, 143 / 145, 145 / 156, 211 / 266
  const bool few = p->synth == KL_SYNTH_AUTO && (size_t)nclips * p->nsets * g.Ly <= 64 * 128;
  const bool tca = p->vjp_tc && p->synth != KL_SYNTH_CUDA_CORES && !few &&
                   (((uintptr_t)targets | (uintptr_t)images) & 15) == 0;
  rc = tca ? kl::vjp_tc_launch(g, p->T, p->ty, nclips, p->nsets, p->bhi, p->blo, p->thi, p->tlo, targets, alpha,
                               threshold, images, loss, p->gpart, p->status, st)
           : kl::vjp_launch_inverse(g, p->tx, p->ty, p->T, nclips, p->nsets, targets, alpha, threshold, images,
                                    loss, p->gpart, st);
  if (rc) return rc;
  const int ns2 = adjoint_split(p, nclips * p->nsets);
  if ((rc = kl::adjoint_launch(p->sg, p->partial, g.nS, 1.0f / ((float)g.Lx * (float)g.Ly), p->gpart, g.nS,
                               nclips * p->nsets, p->HT, p->lam, p->K, p->nsets, ns2, p->gamma, p->gam, st)))
    return rc;
  if ((rc = kl::adjoint_gradient(p->sg, p->gam, nclips, p->nsets * adjoint_parts(p, ns2), 2 * g.Ny, g.ntx, g.ntx, 1, p->Tg,
                                 st)))
    return rc;
  // the gradient is a band-limited synthesis like the image
  const bool tcg = p->bhi && p->synth != KL_SYNTH_CUDA_CORES && !few && kl::synth_tc_aligned(grad);
  rc = tcg ? kl::synth_tc_launch(g, p->Tg, p->ty, p->bhi, p->blo, nclips, grad, p->status, st)
           : kl::socs_launch_inverse(g, p->tx, p->ty, p->Tg, nclips, 1, grad, st);
  if (rc) return rc;
  p->last_vjp_clips = nclips;
  return KL_OK;
}

int kl_socs_set_synthesis(kl_socs_plan p, int mode) {
  KL_CHECK_ARG(p != nullptr, "kl_socs_set_synthesis: plan is NULL");
  KL_CHECK_ARG(mode == KL_SYNTH_AUTO || mode == KL_SYNTH_CUDA_CORES || mode == KL_SYNTH_TENSOR_CORES,
               "kl_socs_set_synthesis: mode must be KL_SYNTH_AUTO, KL_SYNTH_CUDA_CORES or KL_SYNTH_TENSOR_CORES");
  if (mode == KL_SYNTH_TENSOR_CORES && !p->bhi) {
    kl::set_error(p->gen ? "kl_socs_set_synthesis: the general pipeline has no tensor-core synthesis"
                         : "kl_socs_set_synthesis: the tensor-core synthesis needs Lx, Ly multiples of 128 and "
                           "2(2Nx+1) <= 128");
    return KL_ERR_UNSUPPORTED;
  }
  p->synth = mode;
  return KL_OK;
}

int kl_socs_synthesis(kl_socs_plan p, int nclips) {
  if (!p) return KL_ERR_INVALID;
  return use_tc_synthesis(p, nclips) ? KL_SYNTH_TENSOR_CORES : KL_SYNTH_CUDA_CORES;
}

int kl_socs_plan_status(kl_socs_plan p) {
  KL_CHECK_ARG(p != nullptr, "kl_socs_plan_status: plan is NULL");
  KL_CUDA_TRY(cudaDeviceSynchronize());
  if (!p->status) return KL_OK;
  int code = 0;
  KL_CUDA_TRY(cudaMemcpy(&code, p->status, sizeof(int), cudaMemcpyDeviceToHost));
  if (!code) return KL_OK;
  KL_CUDA_TRY(cudaMemset(p->status, 0, sizeof(int)));
  kl::set_error("tensor-core synthesis: pipeline wait timed out (code " + std::to_string(code) + ")");
  return KL_ERR_CUDA;
}

int kl_socs_plan_destroy(kl_socs_plan plan) {
  free_plan(plan);
  return KL_OK;
}

int kl_socs_set_kernels(kl_socs_plan p, int set, const float* re, const float* im,
                        const float* scales) {
  KL_CHECK_ARG(p && re && im && scales, "kl_socs_set_kernels: NULL argument");
  KL_CHECK_ARG(set >= 0 && set < p->nsets, "kl_socs_set_kernels: set out of range");
  return upload_kernels(p, set, re, im, scales);
}

int kl_socs_set_kernels_c64(kl_socs_plan p, int set, const float* krn, const float* scales) {
  KL_CHECK_ARG(p && krn && scales, "kl_socs_set_kernels_c64: NULL argument");
  KL_CHECK_ARG(set >= 0 && set < p->nsets, "kl_socs_set_kernels_c64: set out of range");
  return upload_kernels(p, set, krn, nullptr, scales);
}

int kl_socs_set_kernels_device(kl_socs_plan p, int set, const float2* H_dev, const float* lam_dev,
                               cudaStream_t st) {
  KL_CHECK_ARG(p && H_dev && lam_dev, "kl_socs_set_kernels_device: NULL argument");
  KL_CHECK_ARG(set >= 0 && set < p->nsets, "kl_socs_set_kernels_device: set out of range");
  const size_t nb2 = (size_t)p->g.nby * p->g.nbx, k0 = (size_t)set * p->K;
  if (p->H)
    KL_CUDA_TRY(cudaMemcpyAsync(p->H + k0 * nb2, H_dev, sizeof(float2) * nb2 * p->K, cudaMemcpyDeviceToDevice, st));
  if (int rc = kl::spec_columns(p->sg, H_dev, p->K, p->HT + k0 * kl::spec_kernel_elems(p->sg), st)) return rc;
  KL_CUDA_TRY(cudaMemcpyAsync(p->lam + k0, lam_dev, sizeof(float) * p->K, cudaMemcpyDeviceToDevice, st));
  return KL_OK;
}

int kl_socs_forward(kl_socs_plan p, const float* masks, int nclips, float* images, void* stream) {
  KL_CHECK_ARG(p && masks && images, "kl_socs_forward: NULL argument");
  KL_CHECK_ARG(nclips >= 0 && nclips <= p->max_clips, "kl_socs_forward: nclips exceeds the plan");
  return run_forward(p, masks, nclips, images, (cudaStream_t)stream);
}

int kl_socs_forward_host(kl_socs_plan p, const float* masks_host, int nclips, float* images_host,
                         void* stream) {
  KL_CHECK_ARG(p && masks_host && images_host, "kl_socs_forward_host: NULL argument");
  KL_CHECK_ARG(nclips >= 0 && nclips <= p->max_clips, "kl_socs_forward_host: nclips exceeds the plan");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t px = (size_t)p->g.Lx * p->g.Ly;
  if (p->stage_clips < (size_t)nclips) {
    cudaFree(p->stage_in);
    cudaFree(p->stage_out);
    p->stage_in = p->stage_out = nullptr;
    p->stage_clips = 0;
    int rc;
    if ((rc = alloc((void**)&p->stage_in, sizeof(float) * px * nclips, "mask staging")) ||
        (rc = alloc((void**)&p->stage_out, sizeof(float) * px * nclips * p->nsets, "image staging")))
      return rc;
    p->stage_clips = (size_t)nclips;
  }
  if (nclips == 0) return KL_OK;
  // chunks flow through three streams: copy-in, compute (in order, so the
  // plan's scratch is reused safely), copy-out; the two copy directions and
  // the kernels of neighbouring chunks overlap
  if (!p->hs[0]) {
    for (int i = 0; i < 3; ++i) {
      KL_CUDA_TRY(cudaStreamCreateWithFlags(&p->hs[i], cudaStreamNonBlocking));
      KL_CUDA_TRY(cudaEventCreateWithFlags(&p->hev[i], cudaEventDisableTiming));
    }
  }
  cudaStream_t sin = p->hs[0], scomp = p->hs[1], sout = p->hs[2];
  KL_CUDA_TRY(cudaEventRecord(p->hev[0], st));  // after earlier work on the caller's stream
  for (int i = 0; i < 3; ++i) KL_CUDA_TRY(cudaStreamWaitEvent(p->hs[i], p->hev[0], 0));
  // chunks of about 64 MB of images (up to 16): the copy-out stream idles only
  // while the first chunk is copied in and imaged, and the last copied out
  const size_t outpx = px * p->nsets;
  const size_t outbytes = sizeof(float) * outpx * (size_t)nclips;
  const int nchunks = (int)std::min<size_t>({(size_t)16, std::max<size_t>(1, outbytes >> 26), (size_t)nclips});
  for (int c = 0; c < nchunks; ++c) {
    const int a = (int)((long long)nclips * c / nchunks), b = (int)((long long)nclips * (c + 1) / nchunks);
    if (b == a) continue;
    KL_CUDA_TRY(cudaMemcpyAsync(p->stage_in + px * a, masks_host + px * a, sizeof(float) * px * (b - a),
                                cudaMemcpyHostToDevice, sin));
    KL_CUDA_TRY(cudaEventRecord(p->hev[1], sin));
    KL_CUDA_TRY(cudaStreamWaitEvent(scomp, p->hev[1], 0));
    int rc = run_forward(p, p->stage_in + px * a, b - a, p->stage_out + outpx * a, scomp);
    if (rc) return rc;
    KL_CUDA_TRY(cudaEventRecord(p->hev[2], scomp));
    KL_CUDA_TRY(cudaStreamWaitEvent(sout, p->hev[2], 0));
    KL_CUDA_TRY(cudaMemcpyAsync(images_host + outpx * a, p->stage_out + outpx * a, sizeof(float) * outpx * (b - a),
                                cudaMemcpyDeviceToHost, sout));
  }
  KL_CUDA_TRY(cudaEventRecord(p->hev[0], sout));
  KL_CUDA_TRY(cudaStreamWaitEvent(st, p->hev[0], 0));
  KL_CUDA_TRY(cudaStreamSynchronize(st));
  return p->status ? kl_socs_plan_status(p) : KL_OK;
}

int kl_socs_enable_timing(kl_socs_plan p, int enable) {
  KL_CHECK_ARG(p, "kl_socs_enable_timing: NULL plan");
  p->timing = enable != 0;
  if (!p->timing) drop_events(p);
  return KL_OK;
}

int kl_socs_stage_times(kl_socs_plan p, double* ms, int* launches) {
  KL_CHECK_ARG(p && ms && launches, "kl_socs_stage_times: NULL argument");
  for (int i = 0; i < 3; ++i) {
    ms[i] = 0.0;
    launches[i] = 0;
  }
  for (size_t b = 0; b + 3 < p->events.size(); b += 4) {
    KL_CUDA_TRY(cudaEventSynchronize(p->events[b + 3]));
    for (int i = 0; i < 3; ++i) {
      float t = 0.f;
      KL_CUDA_TRY(cudaEventElapsedTime(&t, p->events[b + i], p->events[b + i + 1]));
      ms[i] += t;
      launches[i] += 1;
    }
  }
  drop_events(p);
  return KL_OK;
}

int kl_mask_spectrum(kl_socs_plan p, const float* masks, int nclips, float* band, void* stream) {
  KL_CHECK_ARG(p && masks && band, "kl_mask_spectrum: NULL argument");
  KL_CHECK_ARG(nclips >= 0 && nclips <= p->max_clips, "kl_mask_spectrum: nclips exceeds the plan");
  cudaStream_t st = (cudaStream_t)stream;
  if (p->gen) {
    const kl::GenGeom& g = p->gg;
    const int nparts = kl::gen_choose_parts(g, nclips, g.nf);
    int rc = kl::gen_launch_rowfwd(g, p->gtab, masks, nclips * g.Ly, p->R, st);
    if (!rc)
      rc = kl::gen_launch_colfwd(g, p->gtab, p->R, nclips, g.nf, g.Ny, 1.0f / ((float)g.Lx * (float)g.Ly), nparts,
                                 p->band, st);
    if (!rc) rc = kl::gen_launch_bandout(g, p->band, nparts, nclips, reinterpret_cast<float2*>(band), st);
    return rc;
  }
  int rc = kl::socs_launch_forward(p->g, p->tx, p->ty, masks, nclips, p->partial, st);
  if (rc) return rc;
  return kl::socs_launch_band(p->g, p->partial, nclips, reinterpret_cast<float2*>(band), st);
}

int kl_fp64_socs_forward(const float* masks, int nclips, int Lx, int Ly, int Nx, int Ny, const float* kernels,
                         const float* scales, int nk, double* images, void* stream) {
  return kl::f64::socs_forward(masks, nclips, Lx, Ly, Nx, Ny, reinterpret_cast<const float2*>(kernels), scales,
                               nk, images, (cudaStream_t)stream);
}

int kl_fp64_socs_vjp(const float* masks, const float* targets, int nclips, int Lx, int Ly, int Nx, int Ny,
                     const float* kernels, const float* scales, int nk, double alpha, double threshold,
                     double* images, double* grad, double* loss, void* stream) {
  return kl::f64::socs_vjp(masks, targets, nclips, Lx, Ly, Nx, Ny, reinterpret_cast<const float2*>(kernels), scales,
                           nk, alpha, threshold, images, grad, loss, (cudaStream_t)stream);
}

int kl_fp64_mask_spectrum(const float* mask, int Lx, int Ly, double* spectrum, void* stream) {
  return kl::f64::mask_spectrum(mask, Lx, Ly, reinterpret_cast<double2*>(spectrum), (cudaStream_t)stream);
}

}  // extern "C"
