// socs_gen.cu -- fused single-precision SOCS imaging for any clip period and
// bands up to a 256-point spectral grid (sm_100a).
//
// Same model as socs_fast.cu -- the K-Litho SOCS image
//     image = sum_k lambda_k |IFFT(H_k . FT(m))|^2 , Fourier-interpolated to Lx x Ly
// (K-Litho-SOCS/klitho_socs.cpp:196-241 calcSOCS, :158-194 FI, fed by
// FT_r2c :70-121) -- but with no restriction on Lx, Ly (the reference takes
// any period, klitho_socs.cpp:256-270) and with spectral grids up to G = 256
// (4N+1 <= 256: 4096^2 clips at NA 1.35 have N = 53, 4N+1 = 213).  The K
// coherent fields and the full-size spectrum never reach HBM.  Stages:
//
//  row_fwd   (HBM-bound) each warp turns mask rows into their Nx+1 row bins:
//            lane l' holds pixels x = l' + Vf i, a real DFT of length Pf over i
//            in registers, then the bins are gathered by the lanes that own
//            them through a per-warp shared buffer (no warp reduce-scatter, so
//            the register count does not grow with the band).
//  col_fwd   the row bins' DFT along y, kept for |fy| <= Ny: 32-point warp FFTs
//            over strips of 32 rows spaced Ly/32 apart when 32 divides Ly,
//            otherwise blocks of 32 rows by one table; strips are split over `nparts` partial bands.
//  spectral  (spectral.cu) the band's K fields, their lambda |E|^2 and its
//            spectrum T, on chip.
//  col_inv   T's columns synthesised along y for every image row (a strip's
//            32-point FFT per thread, or the blocks), giving the rows' coefficients Q[y][b], b <= 2Nx.
//  row_inv   each warp synthesises image rows from Q: lane l'
//            accumulates the Hermitian half of its P sub-bins and runs one
//            length-P complex-to-real transform in registers.
//
// Twiddle tables that depend on the period are made once per plan with exact
// double-precision arguments.  Only row bins (Nx+1 or 2Nx+1 per row), band
// partials and T pass through global memory.
#include <algorithm>
#include <climits>

#include "fft32.cuh"
#include "kl_device.cuh"
#include "kl_internal.h"
#include "kl_launch.cuh"
#include "row_fold.cuh"

namespace kl {

namespace {
constexpr int kT = 256;
constexpr int kW = kT / 32;
constexpr int kSMs = 148;

__host__ __device__ inline int pow2_ge(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}
__device__ __forceinline__ int brev5(int lane) { return (int)(__brev((unsigned)lane) >> 27); }
__device__ __forceinline__ int mod_pos(int a, int m) {
  int r = a % m;
  return r < 0 ? r + m : r;
}

// table offsets inside one float2 buffer
__host__ __device__ inline size_t off_twl(const GenGeom& g) { return (size_t)g.NBX * 32; }
__host__ __device__ inline size_t off_tw2(const GenGeom& g) { return (size_t)g.NBX * 64; }
__host__ __device__ inline size_t off_rly(const GenGeom& g) { return (size_t)g.NBX * 64 + (size_t)g.nC * g.NBX; }
}  // namespace

// ---------------------------------------------------------------------------
// geometry and plan-time tables
// ---------------------------------------------------------------------------
int gen_geometry(int Lx, int Ly, int Nx, int Ny, GenGeom* out) {
  if (Lx <= 0 || Ly <= 0 || Nx < 0 || Ny < 0) {
    set_error("gen_geometry: invalid sizes");
    return KL_ERR_INVALID;
  }
  GenGeom g{};
  g.Lx = Lx;
  g.Ly = Ly;
  g.Nx = Nx;
  g.Ny = Ny;
  g.nbx = 2 * Nx + 1;
  g.nby = 2 * Ny + 1;
  g.nf = Nx + 1;
  g.ntx = 2 * Nx + 1;
  g.nty = 4 * Ny + 1;
  const int gmin = 4 * std::max(Nx, Ny) + 1;
  g.G = std::max(32, pow2_ge(gmin));
  if (g.G > 256) {
    set_error("SOCS path supports 4*max(Nx,Ny)+1 <= 256 (got " + std::to_string(gmin) + ")");
    return KL_ERR_UNSUPPORTED;
  }
  g.RG = g.G / 32;
  // the reference's half-spectrum bookkeeping in FI assumes the SOCS grid
  // 4N+1 fits in half the period; physical optics always satisfies it
  if (4 * Nx + 1 > Lx / 2 || 4 * Ny + 1 > Ly / 2) {
    set_error("band too wide for the clip size (4N+1 must not exceed half the period)");
    return KL_ERR_UNSUPPORTED;
  }
  // synthesis: the largest power of two P <= 64 dividing Lx that leaves at
  // least 32 lanes of work per row
  int P = 1;
  while (P < 64 && Lx % (2 * P) == 0 && Lx / (2 * P) >= 32) P *= 2;
  g.P = P;
  g.V = Lx / P;
  g.Pf = std::min(P, 32);
  g.Vf = Lx / g.Pf;
  g.nC = (std::max(g.V, g.Vf) + 31) / 32;
  const int q = std::max(32, P);
  g.NBX = (g.ntx + q - 1) / q * q;
  g.ystrip = (Ly % 32 == 0) ? 1 : 0;
  g.nS = g.ystrip ? Ly / 32 : (Ly + 31) / 32;
  g.dx = 2 * ((Lx + 1) / 2) - Lx;
  g.dy = 2 * ((Ly + 1) / 2) - Ly;
  *out = g;
  return KL_OK;
}

size_t gen_rowbins_bytes(const GenGeom& g, int nimg, int nbins) {
  return sizeof(float2) * (size_t)nimg * g.Ly * nbins;
}
size_t gen_band_bytes(const GenGeom& g, int n, int nparts, int nrows, int ncols) {
  (void)g;
  return sizeof(float2) * (size_t)n * nparts * nrows * ncols;
}
size_t gen_table_elems(const GenGeom& g) { return off_rly(g) + (size_t)g.Ly + g.Lx; }
const float2* gen_roots_x(const GenGeom& g, const float2* tables) { return tables + off_rly(g) + g.Ly; }

int gen_choose_split(const GenGeom& g, int nimg, int K) {
  // kernel slices per image: the count whose CTAs fill the GPU's resident
  // slots most evenly (waves x work per CTA), with slices of at least 3 kernels
  const long long slots = kSMs, ctas = (long long)g.RG * nimg;
  int best = 1;
  double best_t = 1e30;
  for (int ns = 1; ns <= kGenMaxSplit && (ns == 1 || K / ns >= 3); ns *= 2) {
    const double t = (double)((ctas * ns + slots - 1) / slots) / ns;
    if (t < best_t * 0.98) {
      best_t = t;
      best = ns;
    }
  }
  return best;
}

int gen_choose_parts(const GenGeom& g, int n, int ncols) {
  // enough CTAs of the column transform to cover the GPU, at least 4 strips each; of
  // the blocked one once, at least 2 blocks of rows each
  int np = 1;
  if (!g.ystrip) {
    const int cols = (ncols + 15) / 16;
    while (cols * n * np < kSMs && g.nS / (2 * np) >= 2) np *= 2;
    return np;
  }
  const int groups = (ncols + kW - 1) / kW;
  while (groups * n * np < 2 * kSMs && g.nS / (2 * np) >= 4) np *= 2;
  return np;
}

// twb[b][l] = twl[l][b] = e^{+2 pi i b l / Lx}; tw2[c][b] = e^{+2 pi i b 32 c / Lx};
// rly[m] = e^{+2 pi i m / Ly}; rlx[m] = e^{+2 pi i m / Lx}
__global__ void k_gen_tables(const GenGeom g, float2* __restrict__ t) {
  const size_t n1 = (size_t)g.NBX * 32, n2 = (size_t)g.nC * g.NBX;
  const size_t n = off_rly(g) + g.Ly + g.Lx;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float2 v;
    if (i < n1) {
      const int b = (int)(i / 32), l = (int)(i % 32);
      v = expi2pi_frac((long long)b * l, g.Lx);
    } else if (i < 2 * n1) {
      const size_t j = i - n1;
      const int l = (int)(j / g.NBX), b = (int)(j % g.NBX);
      v = expi2pi_frac((long long)b * l, g.Lx);
    } else if (i < 2 * n1 + n2) {
      const size_t j = i - 2 * n1;
      const int c = (int)(j / g.NBX), b = (int)(j % g.NBX);
      v = expi2pi_frac((long long)b * 32 * c, g.Lx);
    } else if (i < off_rly(g) + g.Ly) {
      v = expi2pi_frac((long long)(i - off_rly(g)), g.Ly);
    } else {
      v = expi2pi_frac((long long)(i - off_rly(g) - g.Ly), g.Lx);
    }
    t[i] = v;
  }
}

namespace {
template <typename Kern>
int set_smem(Kern k, size_t bytes) {
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) {
      set_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
      return KL_ERR_CUDA;
    }
  }
  return KL_OK;
}
int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string(what) + ": " + cudaGetErrorString(e));
    return KL_ERR_CUDA;
  }
  return KL_OK;
}
}  // namespace

int gen_build_tables(const GenGeom& g, float2* tables, cudaStream_t st) {
  const size_t n = gen_table_elems(g);
  const int blocks = (int)std::min<size_t>((n + 255) / 256, 4096);
  k_gen_tables<<<blocks, 256, 0, st>>>(g, tables);
  return check_launch("k_gen_tables");
}

// ---------------------------------------------------------------------------
// 1. row_fwd: rows of `src` (Lx floats each) -> R[row][fx], fx < nbins
// ---------------------------------------------------------------------------
template <int PF>
__global__ void __launch_bounds__(kT) k_gen_rowfwd(const float* src, int nrows, const GenGeom g,
                                                   const float2* __restrict__ tables, int nbins,
                                                   float2* __restrict__ R) {
  constexpr int HS = PF / 2 + 1;
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* tl = reinterpret_cast<float2*>(smem4);  // [32][NBX]  e^{+2 pi i b l / Lx}
  float2* sb = tl + 32 * g.NBX + warp * HS * 33;  // [HS][33]   the lanes' real-DFT outputs
  const float2* twl = tables + off_twl(g);
  const float2* tw2 = tables + off_tw2(g);
  for (int i = threadIdx.x; i < 32 * g.NBX; i += kT) tl[i] = __ldg(twl + i);
  dep_wait();
  dep_launch();
  __syncthreads();
  const int V = g.Vf, nch = (V + 31) / 32, nt = (nbins + 31) / 32;
  for (int row = blockIdx.x * kW + warp; row < nrows; row += gridDim.x * kW) {
    const float* rp = src + (size_t)row * g.Lx;
    float2 acc[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int c = 0; c < nch; ++c) {
      const int lp = lane + 32 * c;
      float val[PF];
      if (lp < V) {
#pragma unroll
        for (int i = 0; i < PF; ++i) val[i] = __ldcs(rp + lp + V * i);
      } else {
#pragma unroll
        for (int i = 0; i < PF; ++i) val[i] = 0.f;
      }
      float2 S[HS];
      rdft_any<PF>(val, S);
#pragma unroll
      for (int k = 0; k < HS; ++k) sb[k * 33 + lane] = S[k];
      __syncwarp();
      // bin fx = sum over the chunk's lanes l of S_l[fx mod PF] e^{-2 pi i fx (l + 32c)/Lx}
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int fx = lane + 32 * t;
        if (t < nt && fx < nbins) {
          const int k = fx % PF;
          const bool cj = 2 * k > PF;
          const int kk = cj ? PF - k : k;
          const float sg = cj ? -1.f : 1.f;
          float2 s = make_float2(0.f, 0.f);
#pragma unroll 8
          for (int l = 0; l < 32; ++l) {
            const float2 sv = sb[kk * 33 + l];
            const float svy = sg * sv.y;
            const float2 w = tl[l * g.NBX + fx];
            s.x = fmaf(sv.x, w.x, fmaf(svy, w.y, s.x));
            s.y = fmaf(svy, w.x, fmaf(-sv.x, w.y, s.y));
          }
          acc[t] = cfma(s, cconj(__ldg(tw2 + (size_t)c * g.NBX + fx)), acc[t]);
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int fx = lane + 32 * t;
      if (t < nt && fx < nbins) R[(size_t)row * nbins + fx] = acc[t];
    }
  }
}

// ---------------------------------------------------------------------------
// 2. col_fwd: R[n][y][fx] -> band[n][part][fy + Yb][fx], |fy| <= Yb, times scale;
// periods of strips (Ly a multiple of 32)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kT) k_gen_colfwd(const float2* R, int ncols, int Yb,
                                                   const GenGeom g, const float2* __restrict__ rly,
                                                   float scale, float2* __restrict__ band) {
  constexpr int MT = 8;  // 2 Yb + 1 <= 256
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fx = blockIdx.x * kW + warp;
  const int n = blockIdx.y, part = blockIdx.z, nparts = gridDim.z;
  dep_wait();
  dep_launch();
  if (fx >= ncols) return;  // whole warp; no block-wide barrier below
  const int nyo = 2 * Yb + 1, Ly = g.Ly;
  const float2* Rn = R + (size_t)n * Ly * ncols;
  float2* out = band + ((size_t)n * nparts + part) * nyo * ncols;
  float2 acc[MT];
#pragma unroll
  for (int t = 0; t < MT; ++t) acc[t] = make_float2(0.f, 0.f);
  const int nS = g.nS;
  const int s0 = (int)((long long)nS * part / nparts), s1 = (int)((long long)nS * (part + 1) / nparts);
  WarpFFT<1, -1> wf;
  wf.init(lane);
  const int q = brev5(lane);
  const int fy0 = q - 32 * ((q + Yb) / 32);  // smallest fy >= -Yb with fy = q (mod 32)
  // the next strip's row bin and phases are loaded while this strip is transformed
  float2 rn = make_float2(0.f, 0.f), pn[MT];
  auto fetch = [&](int s) {
    rn = Rn[(size_t)(s + nS * lane) * ncols + fx];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      const int fy = fy0 + 32 * t;
      pn[t] = fy <= Yb ? __ldg(rly + mod_pos(fy * s, Ly)) : make_float2(1.f, 0.f);
    }
  };
  if (s0 < s1) fetch(s0);
  for (int s = s0; s < s1; ++s) {
    float2 v[1] = {rn};
    float2 p[MT];
#pragma unroll
    for (int t = 0; t < MT; ++t) p[t] = pn[t];
    if (s + 1 < s1) fetch(s + 1);
    wf.run(v, lane);
#pragma unroll
    for (int t = 0; t < MT; ++t) {
      const int fy = fy0 + 32 * t;
      if (fy <= Yb) acc[t] = cfma(v[0], cconj(p[t]), acc[t]);
    }
  }
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    const int fy = fy0 + 32 * t;
    if (fy <= Yb) out[(size_t)(fy + Yb) * ncols + fx] = cscale(acc[t], scale);
  }
}

// The same for Ly not a multiple of 32: the DFT over y as small matrix products, 32
// rows at a time.  y = 32 s + j: a CTA multiplies the block's rows by e^{-2 pi i fy j/Ly}
// (the same 32 x 64 table for every block) and turns the block's sum by
// e^{-2 pi i fy 32 s/Ly}.  Thread = one column fx, four fy.  One frequency per lane with
// both factors gathered for every row took 102 us for seven 1000 x 744 clips.
__global__ void __launch_bounds__(kT) k_gen_colfwd_blocks(const float2* R, int ncols, int Yb,
                                                          const GenGeom g, const float2* __restrict__ rly, int nparts,
                                                          float scale, float2* __restrict__ band) {
  __shared__ float2 Rt[32][16];
  __shared__ float2 Wt[32][64];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int nyo = 2 * Yb + 1, Ly = g.Ly;
  const int fx0 = blockIdx.x * 16, r0 = blockIdx.y * 64;  // rows r = fy + Yb of the band
  const int n = blockIdx.z / nparts, part = blockIdx.z - n * nparts;
  const int s0 = (int)((long long)g.nS * part / nparts), s1 = (int)((long long)g.nS * (part + 1) / nparts);
  const int nr = min(64, nyo - r0), nq = (nr + 15) / 16;
  for (int i = tid; i < 32 * 64; i += kT) {
    const int j = i >> 6, fy = r0 + (i & 63) - Yb;
    Wt[j][i & 63] = cconj(__ldg(rly + mod_pos(fy * j, Ly)));
  }
  dep_wait();
  dep_launch();
  const float2* Rn = R + (size_t)n * Ly * ncols + fx0 + tx;
  const bool colok = fx0 + tx < ncols;
  float2 next[2];
  auto fetch = [&](int s) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int y = 32 * s + ty + 16 * h;
      next[h] = colok && y < Ly ? Rn[(size_t)y * ncols] : make_float2(0.f, 0.f);
    }
  };
  float2 acc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
  if (s0 < s1) fetch(s0);
  for (int s = s0; s < s1; ++s) {
    Rt[ty][tx] = next[0];
    Rt[ty + 16][tx] = next[1];
    __syncthreads();
    if (s + 1 < s1) fetch(s + 1);
    float2 rot[4], blk[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      rot[q] = cconj(__ldg(rly + mod_pos((r0 + ty + 16 * q - Yb) * (32 * s), Ly)));
      blk[q] = make_float2(0.f, 0.f);
    }
    if (nq > 2) {
#pragma unroll 8
      for (int j = 0; j < 32; ++j) {
        const float2 r = Rt[j][tx];
#pragma unroll
        for (int q = 0; q < 4; ++q) blk[q] = cfma(r, Wt[j][ty + 16 * q], blk[q]);
      }
    } else {
#pragma unroll 8
      for (int j = 0; j < 32; ++j) {
        const float2 r = Rt[j][tx];
#pragma unroll
        for (int q = 0; q < 2; ++q) blk[q] = cfma(r, Wt[j][ty + 16 * q], blk[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = cfma(blk[q], rot[q], acc[q]);
    __syncthreads();
  }
  float2* out = band + ((size_t)n * nparts + part) * nyo * ncols + fx0 + tx;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (colok && ty + 16 * q < nr) out[(size_t)(r0 + ty + 16 * q) * ncols] = cscale(acc[q], scale);
}

// ---------------------------------------------------------------------------
// 3. col_inv: T[img][b][a + A] -> Q[img][y][b] = w_b sum_a T e^{2 pi i a y/Ly}
// ---------------------------------------------------------------------------
// Rows y = s + nS j of strip s: a 32-point transform over j of the terms folded mod 32,
//   v[r] = e^{2 pi i r s/Ly} sum_t e^{2 pi i 32 t s/Ly} T[32 t + r].
// A thread makes one strip of one bin: a term is a shared load and four multiply-adds,
// the transform stays in its registers, and a warp's 32 bins of a row are stored
// together.  FP32 issue and the shared loads bound it.  The CTA keeps the terms of its 32
// bins, transposed, for all its strips.  20 images of 4096 rows, 107 bins, 213 terms:
// 49 us; 117 with one transform spread over a warp's lanes by shuffles.
__host__ __device__ inline int colinv_rows(int A) { return (A + 7) / 8 * 8 + (A + 8) / 8 * 8; }

__global__ void __launch_bounds__(kT, 2) k_gen_colinv(const float2* T, int A, int nbins,
                                                      const GenGeom g, const float2* __restrict__ rly,
                                                      float2* __restrict__ Q, int spw) {
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lda = 2 * A + 1, Ly = g.Ly, nS = g.nS, img = blockIdx.z, b0 = 32 * blockIdx.x;
  const int alo = -((A + 7) / 8 * 8), rows = colinv_rows(A), ahi = alo + rows;
  const int tlo = -((31 - alo) / 32), thi = (ahi - 1) / 32;
  float2* Tt = reinterpret_cast<float2*>(smem4);  // [rows: a = alo + r][33]
  float2* Es = Tt + rows * 33 + warp * 32;        // [32] e^{2 pi i r s/Ly} of this warp's strip
  const float2* Ti = T + (size_t)img * nbins * lda;
  int s = blockIdx.y * kW * spw + warp;
  const int s1 = min(nS, (int)(blockIdx.y + 1) * kW * spw);
  // the next strip's phases: r = lane, and t = tlo + lane
  float2 en = make_float2(0.f, 0.f), fn = en;
  auto fetch = [&](int sn) {
    en = __ldg(rly + lane * sn);
    if (lane <= thi - tlo) fn = __ldg(rly + mod_pos(32 * (tlo + lane) * sn, Ly));
  };
  if (s < s1) fetch(s);
  dep_wait();
  dep_launch();
#pragma unroll 2
  for (int q = 0; q < 4; ++q) {
    const int b = b0 + warp + kW * q;
    const float w = b == 0 ? 1.f : 2.f;
    float2 x[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int i = alo + A + lane + 32 * t;
      x[t] = i >= 0 && i < lda && b < nbins ? Ti[(size_t)b * lda + i] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int t = 0; t < 8; ++t)
      if (lane + 32 * t < rows) Tt[(lane + 32 * t) * 33 + warp + kW * q] = cscale(x[t], w);
  }
  __syncthreads();
  float2* Qi = Q + (size_t)img * Ly * nbins + b0 + lane;
  for (; s < s1; s += kW) {
    const float2 f = fn;
    __syncwarp();
    Es[lane] = en;
    __syncwarp();
    if (s + kW < s1) fetch(s + kW);
    float2 v[32];
#pragma unroll
    for (int r = 0; r < 32; ++r) v[r] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int t = tlo; t <= thi; ++t) {
      const float2 F = make_float2(__shfl_sync(0xffffffffu, f.x, t - tlo), __shfl_sync(0xffffffffu, f.y, t - tlo));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int a = 32 * t + 8 * q;
        if (a >= alo && a < ahi) {
          const float2* row = Tt + (a - alo) * 33 + lane;
#pragma unroll
          for (int r = 0; r < 8; ++r) v[8 * q + r] = cfma(row[r * 33], F, v[8 * q + r]);
        }
      }
    }
    const float4* E4 = reinterpret_cast<const float4*>(Es);
#pragma unroll
    for (int r = 0; r < 32; r += 2) {
      const float4 e = E4[r / 2];
      v[r] = cmul(v[r], make_float2(e.x, e.y));
      v[r + 1] = cmul(v[r + 1], make_float2(e.z, e.w));
    }
    fft32<+1>(v);
    if (b0 + lane < nbins) {
#pragma unroll
      for (int j = 0; j < 32; ++j) Qi[(size_t)(s + nS * j) * nbins] = v[fft32_pos(j)];
    }
  }
}

// The same for Ly not a multiple of 32, by blocks of 32 rows y = 32 s + j: T is turned
// by e^{2 pi i a 32 s/Ly} on its way to shared memory, 32 terms a at a time, and
// multiplied by the 32 x 32 table e^{2 pi i a j/Ly}.  Thread = row j, every eighth bin
// (MB of them) of SB blocks: one table value serves all.  A row per lane with both
// factors gathered for every term took 20 us for 14 images of 1000 x 744.
template <int MB, int SB>
__global__ void __launch_bounds__(kT) k_gen_colinv_blocks(const float2* T, int A, int nbins,
                                                          const GenGeom g, const float2* __restrict__ rly,
                                                          float2* __restrict__ Q) {
  extern __shared__ float4 smem4[];
  float2* Wt = reinterpret_cast<float2*>(smem4);  // [32 a][32 j]
  float2* Tt = Wt + 32 * 32;                      // [SB][32 a][8 MB]; at the end [32 j][nbins]
  constexpr int NB = kW * MB;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lda = 2 * A + 1, Ly = g.Ly, s0 = blockIdx.x * SB, img = blockIdx.y;
  const float2* Ti = T + (size_t)img * nbins * lda;
  float2 acc[SB][MB];
#pragma unroll
  for (int s = 0; s < SB; ++s)
#pragma unroll
    for (int q = 0; q < MB; ++q) acc[s][q] = make_float2(0.f, 0.f);
  float2 ph[SB];  // e^{2 pi i a 32 s/Ly} of this lane's a
#pragma unroll
  for (int s = 0; s < SB; ++s) ph[s] = __ldg(rly + mod_pos((lane - A) * (32 * (s0 + s)), Ly));
  dep_wait();
  dep_launch();
  for (int a0 = 0; a0 < lda; a0 += 32) {
#pragma unroll
    for (int i = threadIdx.x; i < 32 * 32; i += kT) Wt[i] = __ldg(rly + mod_pos((a0 + (i >> 5) - A) * (i & 31), Ly));
    const int a = a0 + lane;
#pragma unroll
    for (int q = 0; q < MB; ++q) {
      const int b = warp + kW * q;
      const float2 t = a < lda && b < nbins ? Ti[(size_t)b * lda + a] : make_float2(0.f, 0.f);
#pragma unroll
      for (int s = 0; s < SB; ++s) Tt[(size_t)(s * 32 + lane) * NB + b] = cmul(t, ph[s]);
    }
#pragma unroll
    for (int s = 0; s < SB; ++s) ph[s] = __ldg(rly + mod_pos((a + 32 - A) * (32 * (s0 + s)), Ly));
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
      const float2 w = Wt[k * 32 + lane];
#pragma unroll
      for (int s = 0; s < SB; ++s)
#pragma unroll
        for (int q = 0; q < MB; ++q) acc[s][q] = cfma(Tt[(size_t)(s * 32 + k) * NB + warp + kW * q], w, acc[s][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int s = 0; s < SB; ++s) {
#pragma unroll
    for (int q = 0; q < MB; ++q) {
      const int b = warp + kW * q;
      if (b < nbins) Tt[lane * nbins + b] = cscale(acc[s][q], b == 0 ? 1.f : 2.f);
    }
    __syncthreads();
    const int y0 = 32 * (s0 + s), n = min(32, Ly - y0) * nbins;
    float2* Qi = Q + ((size_t)img * Ly + y0) * nbins;
    for (int i = threadIdx.x; i < n; i += kT) Qi[i] = Tt[i];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// 4. row_inv: Q[row][b] (b < nbins) -> out[row][x] = Re sum_b Q[b] e^{2 pi i b x/Lx}
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(kT) k_gen_rowinv(const float2* Q, int nbins, int nrows,
                                                   const GenGeom g, const float2* __restrict__ tables,
                                                   float* __restrict__ out) {
  constexpr int HY = P / 2 + 1;
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* tb = reinterpret_cast<float2*>(smem4);  // [NBX][32]  e^{+2 pi i b l / Lx}
  float2* qc = tb + g.NBX * 32 + warp * g.NBX;    // [NBX]      this warp's chunk coefficients
  float2* t2s = tb + g.NBX * 32 + kW * g.NBX;     // [nC][NBX]  chunk twiddles, when they fit
  const int V = g.V, nch = (V + 31) / 32;
  const bool t2_shared = gen_t2_in_smem(g);
  const float2* tw2 = t2_shared ? t2s : tables + off_tw2(g);
  for (int i = threadIdx.x; i < 32 * g.NBX; i += kT) tb[i] = __ldg(tables + i);
  if (t2_shared)
    for (int i = threadIdx.x; i < nch * g.NBX; i += kT) t2s[i] = __ldg(tables + off_tw2(g) + i);
  __syncthreads();
  dep_wait();
  const int nbp = (nbins + P - 1) / P * P;
  // each lane holds the coefficients b = lane + 32 t of its warp's row; the
  // next row's are loaded while the current one is synthesised
  float2 qn[4];
  const int row0 = blockIdx.x * kW + warp, rstep = gridDim.x * kW;
  if (row0 < nrows) gen_load_qrow(Q + (size_t)row0 * nbins, nbins, lane, qn);
  for (int row = row0; row < nrows; row += rstep) {
    float2 q[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) q[t] = qn[t];
    if (row + rstep < nrows) gen_load_qrow(Q + (size_t)(row + rstep) * nbins, nbins, lane, qn);
    float* orow = out + (size_t)row * g.Lx;
#pragma unroll 1
    for (int c = 0; c < nch; ++c) {
      // q_c[b] = Q[b] e^{2 pi i b 32 c / Lx}: the lane twiddle then only depends on the lane
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int b = lane + 32 * t;
        if (b < nbp) qc[b] = b < nbins ? cmul(q[t], tw2[(size_t)c * g.NBX + b]) : make_float2(0.f, 0.f);
      }
      __syncwarp();
      float2 Y[HY];
#pragma unroll
      for (int k = 0; k < HY; ++k) Y[k] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int b0 = 0; b0 < nbp; b0 += P) {
#pragma unroll
        for (int k = 0; k < P; ++k) {
          const float2 q = qc[b0 + k];
          const float2 w = tb[(b0 + k) * 32 + lane];
          if (2 * k <= P) {
            Y[k] = cfma(q, w, Y[k]);
          } else {
            Y[P - k].x = fmaf(q.x, w.x, fmaf(-q.y, w.y, Y[P - k].x));
            Y[P - k].y = fmaf(-q.x, w.y, fmaf(-q.y, w.x, Y[P - k].y));
          }
        }
      }
      float o[P];
      c2r_half<P>(Y, o);
      const int lp = lane + 32 * c;
      if (lp < V) {
#pragma unroll
        for (int i = 0; i < P; ++i) __stcs(orow + lp + V * i, o[i]);
      }
      __syncwarp();
    }
  }
  dep_launch();  // the next call's kernel, see kl_launch.cuh
}

// The same for P >= 8 with the twiddles factored (row_fold.cuh).
template <int P, bool SM>
__global__ void __launch_bounds__(kT) k_gen_rowinv_fold(const float2* Q, int nbins, int nrows,
                                                        const GenGeom g, const float2* __restrict__ rlx,
                                                        float* __restrict__ out) {
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* qs = reinterpret_cast<float2*>(smem4) + warp * g.NBX;  // this warp's row
  float2* tb = reinterpret_cast<float2*>(smem4) + kW * g.NBX;
  const int V = g.V, nch = (V + 31) / 32;
  if (SM) row_fold_tables<P>(rlx, V, threadIdx.x, kT, tb);
  __syncthreads();
  dep_wait();
  const int nbp = (nbins + P - 1) / P * P;
  float2 qn[4];
  const int row0 = blockIdx.x * kW + warp, rstep = gridDim.x * kW;
  if (row0 < nrows) gen_load_qrow(Q + (size_t)row0 * nbins, nbins, lane, qn);
  for (int row = row0; row < nrows; row += rstep) {
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (lane + 32 * t < nbp) qs[lane + 32 * t] = qn[t];
    __syncwarp();
    if (row + rstep < nrows) gen_load_qrow(Q + (size_t)(row + rstep) * nbins, nbins, lane, qn);
    float* orow = out + (size_t)row * g.Lx;
#pragma unroll 1
    for (int c = 0; c < nch; ++c) {
      const int lp = lane + 32 * c;
      float2 Y[P / 2 + 1];
      row_fold<P, SM>(qs, nbins, SM ? tb : rlx, V, lp < V ? lp : 0, Y);
      float o[P];
      c2r_half<P>(Y, o);
      if (lp < V) {
#pragma unroll
        for (int i = 0; i < P; ++i) __stcs(orow + lp + V * i, o[i]);
      }
    }
  }
  dep_launch();  // as above
}

// centred FT_r2c band: M(ky,kx) = D(ky,kx) e^{-2 pi i (ky yh/Ly + kx xh/Lx)}
__global__ void k_gen_bandout(const float2* __restrict__ band, int nparts, const GenGeom g,
                              float2* __restrict__ out) {
  const int clip = blockIdx.x;
  const size_t per = (size_t)g.nby * g.nf;
  const float2* b0 = band + (size_t)clip * nparts * per;
  const int yh = (g.Ly + 1) / 2, xh = (g.Lx + 1) / 2;
  for (int i = threadIdx.x; i < g.nby * g.nbx; i += blockDim.x) {
    const int r = i / g.nbx, cidx = i - r * g.nbx;
    const int ky = r - g.Ny, kx = cidx - g.Nx;
    const size_t src = kx >= 0 ? (size_t)r * g.nf + kx : (size_t)(g.nby - 1 - r) * g.nf - kx;
    float2 v = __ldg(b0 + src);
    for (int p = 1; p < nparts; ++p) v = cadd(v, __ldg(b0 + p * per + src));
    if (kx < 0) v = cconj(v);
    const float2 p1 = expi2pi_frac(-(long long)ky * yh, g.Ly);
    const float2 p2 = expi2pi_frac(-(long long)kx * xh, g.Lx);
    out[(size_t)clip * g.nby * g.nbx + i] = cmul(v, cmul(p1, p2));
  }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
namespace {
int row_grid(int nrows, int per_sm) {
  const int need = (nrows + kW - 1) / kW;
  return std::max(1, std::min(need, kSMs * per_sm));
}

template <int PF>
int launch_rowfwd_t(const GenGeom& g, const float2* tables, const float* src, int nrows, int nbins, float2* R,
                    cudaStream_t st) {
  const size_t sm = sizeof(float2) * ((size_t)32 * g.NBX + (size_t)kW * (PF / 2 + 1) * 33);
  auto kern = k_gen_rowfwd<PF>;
  int rc = set_smem(kern, sm);
  if (rc) return rc;
  KL_CUDA_TRY(launch_dependent(kern, row_grid(nrows, 8), kT, sm, st, src, nrows, g, tables, nbins, R));
  return KL_OK;
}

template <int P>
int launch_rowinv_t(const GenGeom& g, const float2* tables, const float2* Q, int nrows, int nbins, float* out,
                    cudaStream_t st) {
  const size_t sm = sizeof(float2) * ((size_t)32 * g.NBX + (size_t)kW * g.NBX +
                                      (gen_t2_in_smem(g) ? (size_t)g.nC * g.NBX : 0));
  auto kern = k_gen_rowinv<P>;
  int rc = set_smem(kern, sm);
  if (rc) return rc;
  KL_CUDA_TRY(launch_dependent(kern, row_grid(nrows, 8), kT, sm, st, Q, nbins, nrows, g, tables, out));
  return KL_OK;
}

template <int P>
int launch_rowinv_fold(const GenGeom& g, const float2* tables, const float2* Q, int nrows, int nbins, float* out,
                       cudaStream_t st) {
  const bool in_smem = row_fold_in_smem(P, g.V);
  const size_t sm = sizeof(float2) * ((size_t)kW * g.NBX + (in_smem ? row_fold_elems(P, g.V) : 0));
  auto kern = in_smem ? k_gen_rowinv_fold<P, true> : k_gen_rowinv_fold<P, false>;
  int rc = set_smem(kern, sm);
  if (rc) return rc;
  // 2, 3, 4, 6 and 8 CTAs per SM: 7 x 2 images of 1000 x 744 (P = 8) 99, 97, 94, 94, 95 us
  // a call, 20 of 4096^2 (P = 64) 829, 837, 828, 826, 827
  KL_CUDA_TRY(launch_dependent(kern, row_grid(nrows, 4), kT, sm, st, Q, nbins, nrows, g, gen_roots_x(g, tables), out));
  return KL_OK;
}

}  // namespace

int gen_launch_rowfwd(const GenGeom& g, const float2* tables, const float* src, int nrows, float2* R,
                      cudaStream_t st) {
  if (nrows <= 0) return KL_OK;
  if (gen_direct_dft(g)) return row_dft(g, gen_roots_x(g, tables), src, nrows / g.Ly, g.nf, R, st);
  switch (g.Pf) {
    case 1: return launch_rowfwd_t<1>(g, tables, src, nrows, g.nf, R, st);
    case 2: return launch_rowfwd_t<2>(g, tables, src, nrows, g.nf, R, st);
    case 4: return launch_rowfwd_t<4>(g, tables, src, nrows, g.nf, R, st);
    case 8: return launch_rowfwd_t<8>(g, tables, src, nrows, g.nf, R, st);
    case 16: return launch_rowfwd_t<16>(g, tables, src, nrows, g.nf, R, st);
    case 32: return launch_rowfwd_t<32>(g, tables, src, nrows, g.nf, R, st);
  }
  set_error("gen_launch_rowfwd: unsupported row transform length");
  return KL_ERR_UNSUPPORTED;
}

int gen_launch_colfwd(const GenGeom& g, const float2* tables, const float2* R, int n, int ncols, int Yb,
                      float scale, int nparts, float2* band, cudaStream_t st) {
  if (n <= 0) return KL_OK;
  if (2 * Yb + 1 > 256) {
    set_error("gen_launch_colfwd: band taller than 256 rows");
    return KL_ERR_UNSUPPORTED;
  }
  if (!g.ystrip) {
    KL_CUDA_TRY(launch_dependent(k_gen_colfwd_blocks, dim3((ncols + 15) / 16, (2 * Yb + 64) / 64, n * nparts), kT, 0, st, R,
                                 ncols, Yb, g, tables + off_rly(g), nparts, scale, band));
    return KL_OK;
  }
  dim3 grid((ncols + kW - 1) / kW, n, nparts);
  KL_CUDA_TRY(launch_dependent(k_gen_colfwd, grid, kT, 0, st, R, ncols, Yb, g, tables + off_rly(g), scale, band));
  return KL_OK;
}

int gen_launch_colinv(const GenGeom& g, const float2* tables, const float2* T, int nimg, int A,
                      int nbins, float2* Q, cudaStream_t st) {
  if (nimg <= 0) return KL_OK;
  if (!g.ystrip) {
    auto launch = [&](auto kern, int mb, int sb) -> int {
      const size_t sm = sizeof(float2) * (size_t)(32 * 32 + sb * 32 * kW * mb);
      if (int rc = set_smem(kern, sm)) return rc;
      KL_CUDA_TRY(launch_dependent(kern, dim3((g.nS + sb - 1) / sb, nimg), kT, sm, st, T, A, nbins, g,
                                   tables + off_rly(g), Q));
      return KL_OK;
    };
    // bins per thread by the band; several blocks per CTA where that leaves registers
    if (nbins <= 32) return launch(k_gen_colinv_blocks<4, 4>, 4, 4);
    if (nbins <= 64) return launch(k_gen_colinv_blocks<8, 2>, 8, 2);
    return launch(k_gen_colinv_blocks<16, 1>, 16, 1);
  }
  // strips per warp: the number with the least work in the longest chain of CTAs (two per
  // SM), making the CTA's terms costing about as much as a strip
  const int tiles = (nbins + 31) / 32, most = (g.nS + kW - 1) / kW;
  int spw = 1;
  long long best = LLONG_MAX;
  for (int m = 1; m <= most; ++m) {
    const long long ctas = (long long)tiles * nimg * ((most + m - 1) / m);
    const long long t = (ctas + 2 * kSMs - 1) / (2 * kSMs) * (m + 1);
    if (t < best) {
      best = t;
      spw = m;
    }
  }
  const size_t sm = sizeof(float2) * ((size_t)colinv_rows(A) * 33 + kW * 32);
  int rc = set_smem(k_gen_colinv, sm);
  if (rc) return rc;
  dim3 grid(tiles, (g.nS + kW * spw - 1) / (kW * spw), nimg);
  KL_CUDA_TRY(launch_dependent(k_gen_colinv, grid, kT, sm, st, T, A, nbins, g, tables + off_rly(g), Q, spw));
  return KL_OK;
}

int gen_launch_rowinv(const GenGeom& g, const float2* tables, const float2* Q, int nimg, int nbins, float* images,
                      cudaStream_t st) {
  if (nimg <= 0) return KL_OK;
  const int nrows = nimg * g.Ly;
  if (gen_direct_synth(g)) return row_synth(g, gen_roots_x(g, tables), Q, nrows, nbins, images, st);
  switch (g.P) {
    case 1: return launch_rowinv_t<1>(g, tables, Q, nrows, nbins, images, st);
    case 2: return launch_rowinv_t<2>(g, tables, Q, nrows, nbins, images, st);
    case 4: return launch_rowinv_t<4>(g, tables, Q, nrows, nbins, images, st);
    case 8: return launch_rowinv_fold<8>(g, tables, Q, nrows, nbins, images, st);
    case 16: return launch_rowinv_fold<16>(g, tables, Q, nrows, nbins, images, st);
    case 32: return launch_rowinv_fold<32>(g, tables, Q, nrows, nbins, images, st);
    case 64: return launch_rowinv_fold<64>(g, tables, Q, nrows, nbins, images, st);
  }
  set_error("gen_launch_rowinv: unsupported row transform length");
  return KL_ERR_UNSUPPORTED;
}

int gen_launch_bandout(const GenGeom& g, const float2* band, int nparts, int nclips, float2* out,
                       cudaStream_t st) {
  if (nclips <= 0) return KL_OK;
  k_gen_bandout<<<nclips, kT, 0, st>>>(band, nparts, g, out);
  return check_launch("k_gen_bandout");
}

}  // namespace kl
