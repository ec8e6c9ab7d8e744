// Fused collide + stream for one level (the per-level hot path).
//
// Reference semantics (Source/Core/AdvanceLBMAtLevel.cpp:20-386): the level
// step FillPatches f^n into a scratch copy with ghosts, collides the valid
// cells in place (collide_forced with the STORED rho^n, u^n and the new force
// F^n), refreshes periodic / inter-box ghosts with post-collision values,
// writes halfway bounce-back ghosts for user_1 faces, pull-streams into f_new
// and recomputes rho, u with F^n/2.
//
// B200 form: one pass, in level_step.cuh (this file holds the host side, the
// macro, initialisation, derived-field and tagging kernels).  A cell's Q
// populations are loaded once, rho^n and u^n recovered from them
// (bit-identical to the stored macro because the reference computed it from
// the same f^n and F^{n-1}; or read from macro_in), collided, and f*(y,q)
// PUSHED to f_out(y+c_q,q) (wrapping periodic directions).  Populations whose
// pull source is a ghost that nobody pushes from are completed by the owner of
// the destination: bounce-back (f*(x,q_bar)), the pre-collision ghost value
// (physical BC / coarse-fine), or, for a ghost covered by another box of the
// level, that ghost collided in place.  What physical ghosts of layer 1 push
// in (self-fill mode, the reference's FillPatch rules) comes from the ghost
// blocks of the same launch, so the cells' code never evaluates boundary
// formulas.  Traffic per cell: Q loads + Q stores of the storage type (plus
// the force band); no scratch copies.
#include <algorithm>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "ilbm_common.cuh"
#include "step_args.cuh"
#include "step_device.cuh"
#include "step_launch.h"

namespace ilbm {

static thread_local std::string g_err;
void set_error(const std::string &msg) { g_err = msg; }
const char *get_error() { return g_err.c_str(); }
int cuda_fail(cudaError_t e, const char *what) {
  set_error(std::string(what) + ": " + cudaGetErrorString(e));
  return ILBM_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Macro pass (calculateMacroForcing) and equilibrium initialisation
// ---------------------------------------------------------------------------
template <class L, int S>
__device__ __forceinline__ void macro_cell(const StepArgs &a, int i, int j, int k, void *macro_out) {
  using R = typename Store<S>::R;
  const int64_t base = fidx(a, i, j, k);
  R f[L::Q];
#pragma unroll
  for (int q = 0; q < L::Q; ++q) f[q] = ldf<L, S>(a, base, q);
  R Fx, Fy, Fz;
  load_force<L, R>(a, a.force, i, j, k, Fx, Fy, Fz);
  R *mo = static_cast<R *>(macro_out);
  const int64_t m = midx(a, i, j, k);
  if (S == ILBM_STORAGE_F64) {
    double rho, u, v, w;
    moments64<L>(reinterpret_cast<double *>(f), Fx, Fy, Fz, rho, u, v, w);
    mo[m] = rho;
    mo[m + a.ms2] = u;
    mo[m + 2 * a.ms2] = v;
    mo[m + 3 * a.ms2] = w;
  } else {
    float drho, u, v, w;
    moments32<L>(reinterpret_cast<float *>(f), Fx, Fy, Fz, drho, u, v, w);
    mo[m] = 1.0f + drho;
    mo[m + a.ms2] = u;
    mo[m + 2 * a.ms2] = v;
    mo[m + 3 * a.ms2] = w;
  }
}

template <class L, int S>
__global__ void __launch_bounds__(256) k_macro(StepArgs a, int rlo0, int rlo1, int rlo2,
                                               int rhi0, void *macro_out) {
  const int i = rlo0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= rhi0) macro_cell<L, S>(a, i, rlo1 + blockIdx.y, rlo2 + blockIdx.z, macro_out);
}

// the macro pass of several boxes: box n's cells [rlo, rhi] start at block first[n]
constexpr int kMacroThreads = 256;
template <class L, int S>
__global__ void __launch_bounds__(kMacroThreads) k_macro_boxes(const __grid_constant__ StepBoxes p) {
  int n = 0;
  while (n + 1 < p.nbox && blockIdx.x >= p.first[n + 1]) ++n;
  const StepArgs &a = p.a[n];
  const uint32_t c = (blockIdx.x - p.first[n]) * kMacroThreads + threadIdx.x;
  if (c >= a.nvec) return;
  const uint32_t row = fast_div(c, a.dvpr), kk = (L::D == 3) ? fast_div(row, a.dvny) : 0u;
  macro_cell<L, S>(a, a.vx0 + (int)(c - row * a.vpr), a.rlo[1] + (int)(row - kk * a.vny), a.rlo[2] + (int)kk,
                   p.macro_out[n]);
}

// InitEquilibrium, AmrCoreLBM.cpp:2117-2164, over the allocated f box
template <class L, int S>
__global__ void __launch_bounds__(256) k_init_eq(StepArgs a, int ng) {
  using T = typename Store<S>::T;
  const int i = a.lo[0] - ng + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = a.lo[1] - ng + blockIdx.y;
  const int k = (L::D == 3) ? a.lo[2] - ng + blockIdx.z : 0;
  if (i > a.hi[0] + ng) return;
  const int64_t m = midx(a, i, j, k);
  const int64_t b = fidx(a, i, j, k);
  T *f1 = static_cast<T *>(const_cast<void *>(a.f_in));
  T *f2 = static_cast<T *>(a.f_out);
  if (S == ILBM_STORAGE_F64) {
    const double r = fmax(ldm<double>(a.macro_in, m), 1.e-12);
    const double u0 = ldm<double>(a.macro_in, m + a.ms2);
    const double v0 = ldm<double>(a.macro_in, m + 2 * a.ms2);
    const double w0 = (L::D == 3) ? ldm<double>(a.macro_in, m + 3 * a.ms2) : 0.0;
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      const double fe = feq64_3<L>(q, r, u0, v0, w0);
      reinterpret_cast<double *>(f1)[b + q * a.fs2] = fe;
      reinterpret_cast<double *>(f2)[b + q * a.fs2] = fe;
    }
  } else {
    const float r = fmaxf(ldm<float>(a.macro_in, m), 1.e-12f);
    const float u0 = ldm<float>(a.macro_in, m + a.ms2);
    const float v0 = ldm<float>(a.macro_in, m + 2 * a.ms2);
    const float w0 = (L::D == 3) ? ldm<float>(a.macro_in, m + 3 * a.ms2) : 0.0f;
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      const float ge = feqs<L>(q, r - 1.0f, u0, v0, w0);
      Store<S>::store(f1 + b + q * a.fs2, ge, sfac<L, S>(a, q));
      Store<S>::store(f2 + b + q * a.fs2, ge, sfac<L, S>(a, q));
    }
  }
}

template <class L, int S>
__global__ void __launch_bounds__(256) k_band_macro(StepArgs a, int blo0, int blo1, int blo2,
                                                    int bn0, int bn1, int bn2, double *EV,
                                                    double *RHO) {
  const int64_t nb = (int64_t)bn0 * bn1 * bn2;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nb;
       t += (int64_t)gridDim.x * blockDim.x)
    band_macro_cell<L, S>(a, blo0, blo1, blo2, bn0, bn1, nb, t, EV, RHO);
}

// the band cells of a list (band indices): the cells a fixed body's stencils
// reach, which are all that its interpolation and export read
template <class L, int S>
__global__ void __launch_bounds__(256) k_band_macro_list(StepArgs a, int blo0, int blo1, int blo2,
                                                         int bn0, int bn1, int bn2,
                                                         const int64_t *__restrict__ cells,
                                                         int ncells, double *EV, double *RHO) {
  const int64_t nb = (int64_t)bn0 * bn1 * bn2;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < ncells; r += gridDim.x * blockDim.x)
    band_macro_cell<L, S>(a, blo0, blo1, blo2, bn0, bn1, nb, cells[r], EV, RHO);
}

// Band macro of a level held in several boxes (caller-filled ghosts), the
// EulerVel of IBMarkerDF::update_forcing (Source/IBM/IBMarkerDF.cpp:1541-1566)
// followed by its FillBoundary (:702-703): a band cell takes rho, u from the
// box whose valid region holds it; a cell that no box holds (a coarse-fine or
// physical ghost of the level) takes the caller-filled ghost value of the
// first box whose grown arrays reach it; a cell that none reaches gets the
// reference's initial EulerVel, zero velocity (and unit density).
template <class L>
__device__ __forceinline__ bool valid_at(const StepArgs &a, int i, int j, int k) {
  return i >= a.lo[0] && i <= a.hi[0] && j >= a.lo[1] && j <= a.hi[1] &&
         (L::D == 2 || (k >= a.lo[2] && k <= a.hi[2]));
}

// the cell can be read from the box's grown arrays: macro_in grown by
// ngrow_m, else f_in and force_prev grown by the smaller of their widths
template <class L>
__device__ __forceinline__ bool readable_at(const StepArgs &a, int i, int j, int k) {
  const int g[3] = {i, j, k};
#pragma unroll
  for (int d = 0; d < L::D; ++d) {
    const int gm = a.lo[d] - a.mgl[d], gf = a.lo[d] - a.fgl[d];
    const int w = a.macro_in ? gm : min(gm, gf);
    if (g[d] < a.lo[d] - w || g[d] > a.hi[d] + w) return false;
  }
  return true;
}

template <class L, int S>
__global__ void __launch_bounds__(256) k_band_macro_boxes(const StepArgs *__restrict__ args, int nargs,
                                                          int blo0, int blo1, int blo2, int bn0,
                                                          int bn1, int bn2, double *EV, double *RHO) {
  const int64_t nb = (int64_t)bn0 * bn1 * bn2;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nb;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = blo0 + (int)(t % bn0);
    const int j = blo1 + (int)((t / bn0) % bn1);
    const int k = (L::D == 3) ? blo2 + (int)(t / ((int64_t)bn0 * bn1)) : 0;
    int src = -1;
    for (int b = 0; b < nargs && src < 0; ++b)
      if (valid_at<L>(args[b], i, j, k)) src = b;
    for (int b = 0; b < nargs && src < 0; ++b)
      if (readable_at<L>(args[b], i, j, k)) src = b;
    double m4[4] = {1.0, 0.0, 0.0, 0.0};
    if (src >= 0) macro_at<L, S>(args[src], i, j, k, m4);
    EV[t] = m4[1];
    EV[t + nb] = m4[2];
    EV[t + 2 * nb] = (L::D == 3) ? m4[3] : 0.0;
    RHO[t] = m4[0];
  }
}

template <class L, int S>
static int launch_band_macro_boxes(ilbm_ctx *ctx, const StepArgs *d_args, int nargs,
                                   const int *blo, const int *bn, double *EV, double *RHO,
                                   cudaStream_t st) {
  const int64_t nb = (int64_t)bn[0] * bn[1] * bn[2];
  const int blocks = (int)std::min<int64_t>((nb + 255) / 256, 2048);
  k_band_macro_boxes<L, S><<<blocks, 256, 0, st>>>(d_args, nargs, blo[0], blo[1], blo[2], bn[0],
                                                   bn[1], bn[2], EV, RHO);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "band macro launch");
  return ILBM_OK;
}

template <class L, int S>
static int launch_band_macro(ilbm_ctx *ctx, const StepArgs &a, const int *blo, const int *bn,
                             double *EV, double *RHO, cudaStream_t st) {
  const int64_t nb = (int64_t)bn[0] * bn[1] * bn[2];
  const int blocks = (int)std::min<int64_t>((nb + 255) / 256, 2048);
  k_band_macro<L, S><<<blocks, 256, 0, st>>>(a, blo[0], blo[1], blo[2], bn[0], bn[1], bn[2], EV,
                                              RHO);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "band macro launch");
  return ILBM_OK;
}

template <class L, int S>
static int launch_band_macro_list(ilbm_ctx *ctx, const StepArgs &a, const int *blo, const int *bn,
                                  const int64_t *cells, int ncells, double *EV, double *RHO,
                                  cudaStream_t st) {
  if (ncells <= 0) return ILBM_OK;
  const int blocks = std::min((ncells + 255) / 256, 2048);
  k_band_macro_list<L, S><<<blocks, 256, 0, st>>>(a, blo[0], blo[1], blo[2], bn[0], bn[1], bn[2],
                                                   cells, ncells, EV, RHO);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "band macro launch");
  return ILBM_OK;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// The ghost shell's sequence (ghost_push): slab d's cells lie outside the box
// in dimension d (two faces), inside it in the active dimensions below d, on
// the grown range of the other dimensions.  Inactive dimensions (periodic
// with self-filled ghosts) have no slab.
static int ghost_offsets(int D, StepArgs &a) {
  int64_t off = 0;
  for (int d = 0; d < 3; ++d) {
    a.goff[d] = (uint32_t)off;
    if (d >= D || (a.self_fill && a.periodic[d])) continue;
    int64_t s = 2;
    for (int e = 0; e < D; ++e)
      if (e != d) {
        const bool inner = e < d && !(a.self_fill && a.periodic[e]);
        s *= (int64_t)(a.hi[e] - a.lo[e] + 1) + (inner ? 0 : 2);
      }
    off += s;
    if (off > INT32_MAX) {
      set_error("box too large: its ghost shell has 2^31 cells or more");
      return ILBM_ERR_RANGE;
    }
  }
  a.goff[3] = (uint32_t)off;
  return ILBM_OK;
}

static int fill_args(const ilbm_ctx *ctx, const ilbm_box &b, const ilbm_level_params *p,
                     StepArgs &a) {
  std::memset(&a, 0, sizeof(a));
  const int D = ctx->dim;
  for (int d = 0; d < 3; ++d) {
    a.lo[d] = (d < D) ? b.lo[d] : 0;
    a.hi[d] = (d < D) ? b.hi[d] : 0;
    a.fgl[d] = (d < D) ? b.lo[d] - b.ngrow_f : 0;
    a.mgl[d] = (d < D) ? b.lo[d] - b.ngrow_m : 0;
  }
  for (int d = 0; d < 3; ++d) {
    a.rlo[d] = a.lo[d];
    a.rhi[d] = a.hi[d];
  }
  a.use_skip = 0;
  a.fs0 = b.fstride[0];
  a.fs1 = b.fstride[1];
  a.fs2 = b.fstride[2];
  a.ms0 = b.mstride[0];
  a.ms1 = b.mstride[1];
  a.ms2 = b.mstride[2];
  a.f_in = b.f_in;
  a.f_out = b.f_out;
  {
    static const int cx9[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
    static const int cy9[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};
    static const int cx19[19] = {0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0};
    static const int cy19[19] = {0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1};
    static const int cz19[19] = {0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1};
    for (int q = 0; q < ctx->q; ++q) {
      int cx = 0, cy = 0, cz = 0;
      if (ctx->q == 9) { cx = cx9[q]; cy = cy9[q]; }
      else if (ctx->q == 19) { cx = cx19[q]; cy = cy19[q]; cz = cz19[q]; }
      else { cx = Lat<27>::cx(q); cy = Lat<27>::cy(q); cz = Lat<27>::cz(q); }
      const int64_t lo = (int64_t)q * b.fstride[2];
      const int64_t dof = lo + cx + (int64_t)cy * b.fstride[0] + (int64_t)cz * b.fstride[1];
      if (lo > INT32_MAX || dof > INT32_MAX || dof < INT32_MIN) {
        set_error("box too large for 32-bit per-direction offsets (Q * component stride >= 2^31)");
        return ILBM_ERR_RANGE;
      }
      a.loff[q] = (int32_t)lo;
      a.doff[q] = (int32_t)dof;
    }
  }
  a.macro_in = b.macro_in;
  a.force = b.force;
  a.force_prev = b.force_prev;
  const float scale16 = (p && p->f16_scale > 0) ? float(p->f16_scale) : 1024.0f;
  for (int q = 0; q < ctx->q; ++q) {
    const bool half = ctx->storage == ILBM_STORAGE_F16_SCALED;
    a.sf[q] = half ? float(ctx->w[q]) / scale16 : 1.0f;
    a.si[q] = half ? float(1.0 / double(a.sf[q])) : 1.0f;
  }
  if (p) {
    for (int d = 0; d < 3; ++d) {
      a.dlo[d] = (d < D) ? p->domain_lo[d] : 0;
      a.dhi[d] = (d < D) ? p->domain_hi[d] : 0;
      a.periodic[d] = (d < D) ? p->periodic[d] : 0;
      a.bclo[d] = p->bc_lo[d];
      a.bchi[d] = p->bc_hi[d];
      for (int c = 0; c < 4; ++c) {
        a.bvlo[d][c] = p->bc_val_lo[d][c];
        a.bvhi[d][c] = p->bc_val_hi[d][c];
      }
      // never read force outside its allocation
      a.flo[d] = (d < D) ? std::max(p->force_lo[d], b.lo[d] - b.ngrow_m) : 0;
      a.fhi[d] = (d < D) ? std::min(p->force_hi[d], b.hi[d] + b.ngrow_m) : 0;
    }
    a.tau = p->tau;
    a.tau64 = Tau64{p->tau, 1.0 / p->tau, 1.0 - 0.5 / p->tau};
    a.om32 = float(1.0 / p->tau);
    a.omh32 = float(1.0 - 0.5 / p->tau);
    a.self_fill = (p->ghost_mode == ILBM_GHOST_SELF);
    a.use_uniform = p->use_uniform_force;
    for (int d = 0; d < 3; ++d) a.uf[d] = p->uniform_force[d];
    a.f16_scale = scale16;
    // what each face does with the populations that leave through it
    for (int d = 0; d < D; ++d) {
      auto face = [&](bool domain_face, int bc) -> int {
        if (!domain_face) return FACE_BOX;
        if (a.periodic[d]) return a.self_fill ? FACE_WRAP : FACE_PERIODIC;
        return bc == ILBM_BC_USER_1 ? FACE_REFLECT : FACE_PHYS;
      };
      a.face_lo[d] = face(a.lo[d] == a.dlo[d], a.bclo[d]);
      a.face_hi[d] = face(a.hi[d] == a.dhi[d], a.bchi[d]);
    }
    int rc = ghost_offsets(D, a);
    if (rc) return rc;
    if (p->ghost_mode == ILBM_GHOST_CALLER) {
      if (p->nlevel_boxes > kMaxLevelBoxes) {
        set_error("level has more boxes than one call supports (64); split the call");
        return ILBM_ERR_RANGE;
      }
      a.nlb = p->nlevel_boxes;
      if (a.nlb > 0)
        for (int c = 0; c < 6; ++c) a.lb0[c] = p->level_boxes[c];
    }
  } else {
    a.f16_scale = scale16;
  }
  return ILBM_OK;
}

// magic of a division by d (1 <= d < 2^31) of numbers below 2^31 (fast_div):
// n / d = (floor(n m / 2^32) + n) >> l with l = ceil(log2 d) and
// m = floor(2^32 (2^l - d) / d) + 1
DivMagic div_magic(uint32_t d) {
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  DivMagic m;
  m.mul = (uint32_t)(((1ull << 32) * ((1ull << l) - d)) / d + 1);
  m.shift = l;
  return m;
}

// the cells [rlo, rhi] of a launch as a sequence of V-cell vectors; false: empty
bool plan_vectors(StepArgs &a, int dim, int V) {
  const int ny = a.rhi[1] - a.rlo[1] + 1, nz = (dim == 3) ? a.rhi[2] - a.rlo[2] + 1 : 1;
  a.nvec = 0;
  if (a.rhi[0] < a.rlo[0] || ny <= 0 || nz <= 0) return false;
  // the vector form goes by the columns that populations land on: those of
  // the cells and their neighbours inside the box
  const int x0 = V > 1 ? std::max(a.rlo[0] - 1, a.lo[0]) : a.rlo[0];
  const int x1 = V > 1 ? std::min(a.rhi[0] + 1, a.hi[0]) : a.rhi[0];
  a.vx0 = a.lo[0] + (x0 - a.lo[0]) / V * V;
  a.vpr = (uint32_t)((x1 - a.vx0) / V + 1);
  a.vny = (uint32_t)ny;
  a.dvpr = div_magic(a.vpr);
  a.dvny = div_magic(a.vny);
  a.nvec = (uint32_t)((int64_t)a.vpr * ny * nz);
  a.forced = a.force == nullptr && a.force_prev == nullptr && a.use_uniform &&
             (a.uf[0] != 0.0 || a.uf[1] != 0.0 || a.uf[2] != 0.0);
  return true;
}

template <class L, int S>
static int launch_step(ilbm_ctx *ctx, const StepArgs &a) {
  launch_cells<L, S>(ctx, a, ctx->stream, true);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "level step launch");
  return ILBM_OK;
}

// the cells [a.rlo, a.rhi] of a level step, with the ghost-shell push or not
template <class L, int S>
static int launch_step_part(ilbm_ctx *ctx, const StepArgs &a, bool with_ghosts) {
  launch_cells<L, S>(ctx, a, ctx->stream, with_ghosts);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "level step launch");
  return ILBM_OK;
}

// Level step whose band [blo,bhi] waits for `band_ready` (recorded on another
// stream): ghost push and every cell outside the band run first, then the band.
template <class L, int S>
static int launch_step_split(ilbm_ctx *ctx, const StepArgs &a, const int *blo, const int *bhi,
                             cudaEvent_t band_ready) {
  StepArgs outer = a;
  outer.use_skip = 1;
  for (int d = 0; d < 3; ++d) {
    outer.slo[d] = blo[d];
    outer.shi[d] = bhi[d];
  }
  launch_cells<L, S>(ctx, outer, ctx->stream, true);
  cudaError_t e = cudaStreamWaitEvent(ctx->stream, band_ready, 0);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent");
  StepArgs inner = a;
  for (int d = 0; d < 3; ++d) {
    inner.rlo[d] = blo[d];
    inner.rhi[d] = bhi[d];
  }
  launch_cells<L, S>(ctx, inner, ctx->stream, false, true);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "level step launch");
  return ILBM_OK;
}

template <class L, int S>
static int launch_macro(ilbm_ctx *ctx, const StepArgs &a, const int *rlo, const int *rhi,
                        void *macro_out) {
  const int nx = rhi[0] - rlo[0] + 1, ny = rhi[1] - rlo[1] + 1;
  const int nz = (L::D == 3) ? rhi[2] - rlo[2] + 1 : 1;
  if (nx <= 0 || ny <= 0 || nz <= 0) return ILBM_OK;
  const int bx = nx >= 256 ? 256 : ((nx + 31) / 32) * 32;
  dim3 grid((nx + bx - 1) / bx, ny, nz);
  k_macro<L, S><<<grid, bx, 0, ctx->stream>>>(a, rlo[0], rlo[1], (L::D == 3) ? rlo[2] : 0,
                                              rhi[0], macro_out);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "macro launch");
  return ILBM_OK;
}

template <class L, int S>
static int launch_init(ilbm_ctx *ctx, const StepArgs &a, int ng) {
  const int nx = a.hi[0] - a.lo[0] + 1 + 2 * ng, ny = a.hi[1] - a.lo[1] + 1 + 2 * ng;
  const int nz = (L::D == 3) ? a.hi[2] - a.lo[2] + 1 + 2 * ng : 1;
  const int bx = nx >= 256 ? 256 : ((nx + 31) / 32) * 32;
  dim3 grid((nx + bx - 1) / bx, ny, nz);
  k_init_eq<L, S><<<grid, bx, 0, ctx->stream>>>(a, ng);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "init launch");
  return ILBM_OK;
}


static int check_box(const ilbm_ctx *ctx, const ilbm_box &b, bool need_out) {
  if (!b.f_in || (need_out && !b.f_out)) {
    set_error("box: f_in/f_out must be set");
    return ILBM_ERR_ARG;
  }
  for (int d = 0; d < ctx->dim; ++d)
    if (b.hi[d] < b.lo[d]) {
      set_error("box: empty valid region");
      return ILBM_ERR_ARG;
    }
  if (b.fstride[0] <= 0 || b.fstride[1] <= 0 || b.fstride[2] <= 0) {
    set_error("box: f strides must be positive");
    return ILBM_ERR_ARG;
  }
  return ILBM_OK;
}

static int check_params(const ilbm_ctx *ctx, const ilbm_level_params *p) {
  if (!p) {
    set_error("level params missing");
    return ILBM_ERR_ARG;
  }
  if (!(p->tau > 0.5)) {
    set_error("tau must exceed 0.5");
    return ILBM_ERR_ARG;
  }
  for (int d = 0; d < ctx->dim; ++d) {
    if (p->periodic[d]) continue;
    for (int s = 0; s < 2; ++s) {
      const int bc = s ? p->bc_hi[d] : p->bc_lo[d];
      if (bc != ILBM_BC_FOEXTRAP && bc != ILBM_BC_EXT_DIR && bc != ILBM_BC_USER_1 &&
          bc != ILBM_BC_USER_2) {
        set_error("non-periodic face needs BC foextrap(2), ext_dir(3), user_1(1001) or user_2(1002)");
        return ILBM_ERR_UNSUPPORTED;
      }
    }
  }
  return ILBM_OK;
}

// Internal entry for the IB: band macro of box `b` into EV (3 x nb) and RHO.
int band_macro(ilbm_ctx *ctx, const ilbm_box &b, const ilbm_level_params *p, const int *blo,
               const int *bn, double *EV, double *RHO, cudaStream_t st) {
  StepArgs a;
  int rc = fill_args(ctx, b, p, a);
  if (rc) return rc;
  return ILBM_DISPATCH(ctx, launch_band_macro, ctx, a, blo, bn, EV, RHO, st);
}

// Band macro on the listed band cells only.
int band_macro_list(ilbm_ctx *ctx, const ilbm_box &b, const ilbm_level_params *p, const int *blo,
                    const int *bn, const int64_t *cells, int ncells, double *EV, double *RHO,
                    cudaStream_t st) {
  StepArgs a;
  int rc = fill_args(ctx, b, p, a);
  if (rc) return rc;
  return ILBM_DISPATCH(ctx, launch_band_macro_list, ctx, a, blo, bn, cells, ncells, EV, RHO, st);
}

// StepArgs of one box of a level, for kernels that take several boxes
int box_step_args(const ilbm_ctx *ctx, const ilbm_box &b, const ilbm_level_params *p,
                  StepArgs *out) {
  return fill_args(ctx, b, p, *out);
}

// Band macro over several boxes whose StepArgs are in device memory.
int band_macro_boxes(ilbm_ctx *ctx, const StepArgs *d_args, int nargs, const int *blo,
                     const int *bn, double *EV, double *RHO, cudaStream_t st) {
  return ILBM_DISPATCH(ctx, launch_band_macro_boxes, ctx, d_args, nargs, blo, bn, EV, RHO, st);
}

// Level step with the band [blo,bhi] deferred until `band_ready`.
int level_step_split(ilbm_ctx *ctx, const ilbm_box &b, const ilbm_level_params *p,
                     const int *blo, const int *bhi, cudaEvent_t band_ready) {
  StepArgs a;
  int rc = fill_args(ctx, b, p, a);
  if (rc) return rc;
  return ILBM_DISPATCH(ctx, launch_step_split, ctx, a, blo, bhi, band_ready);
}

// ---- internal entries of the batch engine (batch.cu) ----------------------

// StepArgs of one batched case: self-filled ghosts, one box equal to the
// domain, distinct f_in / f_out with a ghost layer, macro recovered from f
// (macro_in is not read: the case has taken its first step already).
int batch_case_args(const ilbm_ctx *ctx, const ilbm_box &b, const ilbm_level_params *p,
                    StepArgs *out) {
  int rc = check_params(ctx, p);
  if (rc) return rc;
  if (p->ghost_mode != ILBM_GHOST_SELF) {
    set_error("batched cases use self-filled ghosts (ILBM_GHOST_SELF)");
    return ILBM_ERR_ARG;
  }
  for (int d = 0; d < ctx->dim; ++d)
    if (b.lo[d] != p->domain_lo[d] || b.hi[d] != p->domain_hi[d]) {
      set_error("batched case: the box must equal the domain");
      return ILBM_ERR_ARG;
    }
  if ((rc = check_box(ctx, b, true))) return rc;
  if (b.ngrow_f < 1 || b.f_in == b.f_out) {
    set_error("batched case: f arrays need a ghost layer and f_in != f_out");
    return ILBM_ERR_ARG;
  }
  if ((b.force || b.force_prev) && (b.mstride[0] <= 0 || b.mstride[1] <= 0 || b.mstride[2] <= 0)) {
    set_error("batched case: force strides must be positive");
    return ILBM_ERR_ARG;
  }
  ilbm_box bb = b;
  bb.macro_in = nullptr;
  bb.macro_out = nullptr;
  if ((rc = fill_args(ctx, bb, p, *out))) return rc;
  out->ghost_blocks = 0;
  return ILBM_OK;
}

// ghost-push chunks of w threads for one case (one ghost cell per thread); 0 when every face is a self-filled periodic one
int batch_ghost_chunks(const ilbm_ctx *, const StepArgs &a, int w) {
  return (int)(((int64_t)a.goff[3] + w - 1) / w);
}

template <class L, int S>
static int vec_width_of(const ilbm_ctx *, const StepArgs &a, int *V) {
  *V = vec_width<L, S>(a);
  return ILBM_OK;
}

uint32_t batch_per_block(int V, int w) { return step_vectors_per_block(V, (uint32_t)w); }

// A batch of few cells in all takes the cell form, as a single small level does
// (prefers_cells): up to 2^16, 2^17 where a case has a reflecting y or z face (B200,
// us per step, vector / cell form: 4 Taylor-Green boxes of 64 x 64 FP32 8.3 / 7.2, 16 of
// them 8.6 / 8.3, 24 9.3 / 8.5, 48 10.3 / 12.4; FP16 9.3 / 8.3, 9.3 / 9.3, 9.3 / 10.3, 10.7 /
// 15.5; 4 channels of 256 x 128 11.4 / 9.3 FP32 and 15.5 / 12.4 FP16, 16 of them 16.5 /
// 16.5 and 21.6 / 20.6, 24 18.5 / 22.6 and 23.9 / 29.8).  args: both buffer parities.
static bool batch_prefers_cells(const ilbm_ctx *ctx, const StepArgs *args, int n) {
  int64_t total = 0;
  bool wall = false;
  for (int c = 0; c < n / 2; ++c) {
    int64_t cells = 1;
    for (int d = 0; d < ctx->dim; ++d) {
      cells *= args[c].rhi[d] - args[c].rlo[d] + 1;
      if (d > 0) wall = wall || args[c].face_lo[d] == FACE_REFLECT || args[c].face_hi[d] == FACE_REFLECT;
    }
    total += cells;
  }
  return total <= (wall ? 1 << 17 : 1 << 16);
}

// the vector sequences of the cases' cells, V cells per vector for all of them
int batch_plan(const ilbm_ctx *ctx, StepArgs *args, int n, int *V) {
  *V = 0;
  for (int c = 0; c < n; ++c) {
    int v = 1, rc = ILBM_DISPATCH(ctx, vec_width_of, ctx, args[c], &v);
    if (rc) return rc;
    *V = (*V == 0) ? v : std::min(*V, v);
  }
  if (batch_prefers_cells(ctx, args, n)) *V = 1;
  for (int c = 0; c < n; ++c) {
    const StepArgs &a = args[c];
    int64_t vectors = (a.rhi[0] - a.rlo[0] + *V) / *V;  // (a self-filled box: its rows start on vectors)
    for (int d = 1; d < ctx->dim; ++d) vectors *= a.rhi[d] - a.rlo[d] + 1;
    if (vectors >= INT32_MAX - 1024) {  // (fast_div, with the tiles' last lanes beyond the end)
      set_error("batched case: fewer than 2^31 vectors of cells (a cell each in unaligned rows)");
      return ILBM_ERR_RANGE;
    }
    plan_vectors(args[c], ctx->dim, *V);
  }
  return ILBM_OK;
}

int batch_step_launch(ilbm_ctx *ctx, const StepArgs *d_args, const StepTile *d_tiles, int ntiles,
                      int V, int w, int blocks, const int *steps, const int *limit, cudaStream_t st) {
  if (ntiles <= 0) return ILBM_OK;
  return ILBM_DISPATCH(ctx, launch_step_batch, ctx, d_args, d_tiles, ntiles, V, w, blocks, steps, limit,
                       st);
}

// resident blocks of w threads per SM for the batched level step
int batch_step_occupancy(const ilbm_ctx *ctx, int V, int w, int *per_sm) {
  return ILBM_DISPATCH(ctx, occupancy_step_batch, ctx, V, w, per_sm);
}

// ---- derived fields and refinement tags ------------------------------------
// UpdateDerivedMacroFields / visPara (Source/Core/AmrCoreLBM.cpp:105-168,
// Source/LBM/visPara.H:10-54): vorticity from central differences of the
// FillPatched velocity (2D: dv/dx - du/dy; 3D: |curl u|) and pressure
// (rho - 1)/3 on valid cells; the band macro over the box grown by one gives
// the ghost values with the FillPatch rules.  Also the level maximum of the
// vorticity (ErrorEst's vortMax, AmrCoreLBM.cpp:1047) as block partials.
struct DeriveArgs {
  int dim;
  int lo[3], hi[3];
  int blo[3], bn[3];
  int64_t nb;
  int mgl[3];
  int64_t ms0, ms1;
  double dx[3];
};

__device__ __forceinline__ double ev_at(const DeriveArgs &d, const double *EV, int c, int i, int j, int k) {
  return EV[(int64_t)c * d.nb + (i - d.blo[0]) + (int64_t)(j - d.blo[1]) * d.bn[0] +
            (int64_t)(k - d.blo[2]) * d.bn[0] * d.bn[1]];
}

template <class R>
__global__ void __launch_bounds__(256) k_derive(DeriveArgs d, const double *EV, const double *RHO,
                                                R *vor, R *pres, double *bmax) {
  __shared__ double sh[8];
  const int nx = d.hi[0] - d.lo[0] + 1, ny = d.hi[1] - d.lo[1] + 1;
  const int nz = (d.dim == 3) ? d.hi[2] - d.lo[2] + 1 : 1;
  const int64_t n = (int64_t)nx * ny * nz;
  double mx = -1.0e300;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = d.lo[0] + (int)(t % nx), j = d.lo[1] + (int)((t / nx) % ny);
    const int k = (d.dim == 3) ? d.lo[2] + (int)(t / ((int64_t)nx * ny)) : 0;
    const double dv_dx = X::div(X::sub(ev_at(d, EV, 1, i + 1, j, k), ev_at(d, EV, 1, i - 1, j, k)),
                                X::mul(2.0, d.dx[0]));
    const double du_dy = X::div(X::sub(ev_at(d, EV, 0, i, j + 1, k), ev_at(d, EV, 0, i, j - 1, k)),
                                X::mul(2.0, d.dx[1]));
    double w;
    if (d.dim == 3) {
      const double du_dz = X::div(X::sub(ev_at(d, EV, 0, i, j, k + 1), ev_at(d, EV, 0, i, j, k - 1)),
                                  X::mul(2.0, d.dx[2]));
      const double dw_dx = X::div(X::sub(ev_at(d, EV, 2, i + 1, j, k), ev_at(d, EV, 2, i - 1, j, k)),
                                  X::mul(2.0, d.dx[0]));
      const double dv_dz = X::div(X::sub(ev_at(d, EV, 1, i, j, k + 1), ev_at(d, EV, 1, i, j, k - 1)),
                                  X::mul(2.0, d.dx[2]));
      const double dw_dy = X::div(X::sub(ev_at(d, EV, 2, i, j + 1, k), ev_at(d, EV, 2, i, j - 1, k)),
                                  X::mul(2.0, d.dx[1]));
      const double ox = X::sub(dw_dy, dv_dz), oy = X::sub(du_dz, dw_dx), oz = X::sub(dv_dx, du_dy);
      w = __dsqrt_rn(X::add(X::add(X::mul(ox, ox), X::mul(oy, oy)), X::mul(oz, oz)));
    } else {
      w = X::sub(dv_dx, du_dy);
    }
    const int64_t m = (int64_t)(i - d.mgl[0]) + (int64_t)(j - d.mgl[1]) * d.ms0 +
                      (int64_t)(k - d.mgl[2]) * d.ms1;
    const int64_t b = (i - d.blo[0]) + (int64_t)(j - d.blo[1]) * d.bn[0] +
                      (int64_t)(k - d.blo[2]) * d.bn[0] * d.bn[1];
    if (vor) vor[m] = R(w);
    if (pres) pres[m] = R(X::div(X::sub(RHO[b], 1.0), 3.0));
    mx = fmax(mx, w);
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = sh[0];
    for (int w2 = 1; w2 < (int)(blockDim.x >> 5); ++w2) t = fmax(t, sh[w2]);
    bmax[blockIdx.x] = t;
  }
}

__global__ void k_max_final(const double *bmax, int nb, double *out) {
  if (threadIdx.x == 0) {
    double t = -1.0e300;
    for (int b = 0; b < nb; ++b) t = fmax(t, bmax[b]);
    *out = t;
  }
}

// ErrorEst tagging (AmrCoreLBM.cpp:1145-1180, Tagging.H:12-18) on valid
// cells: cleared inside the no-refine x zones, set where |vorticity| >
// threshold or inside the body refinement box; tags[i + nx*(j + ny*k)].
struct TagArgs {
  int dim;
  int lo[3], hi[3];
  int mgl[3];
  int64_t ms0, ms1;
  double threshold;
  int use_box;
  double box_lo[3], box_hi[3];
  double nr_lo, nr_hi;
  double plo[3], phi[3], dx[3];
  int use_ls;                  // level-set band of a cylinder / sphere body
  double ls_c[3], ls_r, ls_band;
};

template <class R>
__global__ void __launch_bounds__(256) k_tags(TagArgs g, const R *vor, unsigned char *tags,
                                              unsigned long long *count) {
  const int nx = g.hi[0] - g.lo[0] + 1, ny = g.hi[1] - g.lo[1] + 1;
  const int nz = (g.dim == 3) ? g.hi[2] - g.lo[2] + 1 : 1;
  const int64_t n = (int64_t)nx * ny * nz;
  unsigned long long mine = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = g.lo[0] + (int)(t % nx), j = g.lo[1] + (int)((t / nx) % ny);
    const int k = (g.dim == 3) ? g.lo[2] + (int)(t / ((int64_t)nx * ny)) : 0;
    const double x = X::add(g.plo[0], X::mul(X::add(double(i), 0.5), g.dx[0]));
    unsigned char tag = 0;
    bool blocked = false;
    if (g.nr_lo > 0.0 || g.nr_hi > 0.0)
      blocked = (x <= X::add(g.plo[0], g.nr_lo)) || (x >= X::sub(g.phi[0], g.nr_hi));
    if (!blocked) {
      const int64_t m = (int64_t)(i - g.mgl[0]) + (int64_t)(j - g.mgl[1]) * g.ms0 +
                        (int64_t)(k - g.mgl[2]) * g.ms1;
      if (fabs(double(vor[m])) > g.threshold) tag = 1;
      if (g.use_ls) {
        // signed distance at the cell centre, as LevelSetManager builds it
        const double y = X::add(g.plo[1], X::mul(X::add(double(j), 0.5), g.dx[1]));
        const double ex = X::sub(x, g.ls_c[0]), ey = X::sub(y, g.ls_c[1]);
        double r2 = X::add(X::mul(ex, ex), X::mul(ey, ey));
        if (g.dim == 3) {
          const double z = X::add(g.plo[2], X::mul(X::add(double(k), 0.5), g.dx[2]));
          const double ez = X::sub(z, g.ls_c[2]);
          r2 = X::add(r2, X::mul(ez, ez));
        }
        if (X::sub(__dsqrt_rn(r2), g.ls_r) < g.ls_band) tag = 1;
      }
      if (g.use_box) {
        const double y = X::add(g.plo[1], X::mul(X::add(double(j), 0.5), g.dx[1]));
        const double z = (g.dim == 3) ? X::add(g.plo[2], X::mul(X::add(double(k), 0.5), g.dx[2])) : 0.0;
        if (x >= g.box_lo[0] && x <= g.box_hi[0] && y >= g.box_lo[1] && y <= g.box_hi[1] &&
            z >= g.box_lo[2] && z <= g.box_hi[2])
          tag = 1;
      }
    }
    tags[t] = tag;
    mine += tag;
  }
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(count, mine);
}

template <class L, int S>
static int launch_boxes(ilbm_ctx *ctx, StepBoxes &p, const StepBoxes &whole) {
  if (!launch_step_boxes<L, S>(ctx, p, ctx->stream)) {
    // too many cells together: one launch per box (in slices along the last
    // dimension where it alone is too large), with the level's boxes beside it
    for (int n = 0; n < whole.nbox; ++n) {
      StepBoxes one = whole;
      one.nbox = 1;
      one.a[0] = whole.a[n];
      const int e = L::D - 1, last = one.a[0].rhi[e];
      int64_t slice = 1;  // below 2^28: the offsets of a neighbouring layer fit 32 bits
      for (int d = 0; d < e; ++d) slice *= one.a[0].rhi[d] - one.a[0].rlo[d] + 1;
      const int64_t most = std::max<int64_t>(1, kMaxLaunchCells / slice);
      for (int64_t s = one.a[0].rlo[e]; s <= last; s += most) {
        one.a[0].rlo[e] = (int)s;
        one.a[0].rhi[e] = (int)std::min<int64_t>(last, s + most - 1);
        if (!launch_step_boxes<L, S>(ctx, one, ctx->stream)) {
          set_error("box too large for one launch");
          return ILBM_ERR_RANGE;
        }
        one.a[0].goff[3] = 0;  // the ghost shell goes with the first slice
      }
    }
  }
  return ILBM_OK;
}

template <class L, int S>
static int launch_macro_boxes(ilbm_ctx *ctx, StepBoxes &p) {
  uint32_t blocks = 0;
  for (int n = 0; n < p.nbox; ++n) {
    plan_vectors(p.a[n], L::D, 1);
    p.first[n] = blocks;
    blocks += (p.a[n].nvec + kMacroThreads - 1) / kMacroThreads;
  }
  p.first[p.nbox] = blocks;
  if (blocks == 0) return ILBM_OK;
  k_macro_boxes<L, S><<<blocks, kMacroThreads, 0, ctx->stream>>>(p);
  ctx->launches++;
  return ILBM_OK;
}

// the boxes of a level (caller-filled ghosts, checked): kMaxStepBoxes to a
// launch, then their macro fields
static int level_step_boxes(ilbm_ctx *ctx, const ilbm_box *boxes, int nbox, const ilbm_level_params *p) {
  if (p->nlevel_boxes > kMaxLevelBoxes) {
    set_error("level has more boxes than one call supports (64); split the call");
    return ILBM_ERR_RANGE;
  }
  std::vector<StepBoxes> h(2);  // (the launch's parameters are too large for the stack to be pleasant)
  StepBoxes &s = h[0], &m = h[1];
  std::memset(&s, 0, sizeof(s));
  for (int n = 0; n < p->nlevel_boxes; ++n)
    for (int c = 0; c < 6; ++c) s.lb.lb[n][c] = p->level_boxes[6 * n + c];
  for (int b0 = 0; b0 < nbox; b0 += kMaxStepBoxes) {
    s.nbox = std::min(nbox - b0, kMaxStepBoxes);
    int64_t cells = 0;
    for (int n = 0; n < s.nbox; ++n) {
      int rc = fill_args(ctx, boxes[b0 + n], p, s.a[n]);
      if (rc) return rc;
      int64_t c = 1;
      for (int d = 0; d < ctx->dim; ++d) c *= s.a[n].rhi[d] - s.a[n].rlo[d] + 1;
      cells = std::max(cells, c);
    }
    m = s;
    int rc = ILBM_DISPATCH(ctx, launch_boxes, ctx, m, s);
    if (rc) return rc;
    m = s;
    m.nbox = 0;
    for (int n = 0; n < s.nbox; ++n) {
      const ilbm_box &b = boxes[b0 + n];
      if (!b.macro_out) continue;
      if (cells > (1 << 26)) {  // as above: one launch per box
        StepArgs am = s.a[n];
        am.f_in = b.f_out;
        if ((rc = ILBM_DISPATCH(ctx, launch_macro, ctx, am, am.rlo, am.rhi, b.macro_out))) return rc;
        continue;
      }
      m.a[m.nbox] = s.a[n];
      m.a[m.nbox].f_in = b.f_out;
      m.macro_out[m.nbox++] = b.macro_out;
    }
    if (m.nbox > 0 && (rc = ILBM_DISPATCH(ctx, launch_macro_boxes, ctx, m))) return rc;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "level step launch");
  return ILBM_OK;
}

// one level step; with mlo / mhi the boxes' macro_in holds stored values
// only on [mlo, mhi] (elsewhere rho, u are recovered from f^n and F^{n-1}),
// and macro_out is written there only.  part (one box only): 0 = the whole
// step; 1 = the ghost-shell push and the cells of the first half of the box
// along its last dimension; 2 = the cells of the second half, then
// macro_out.  Every (cell, direction) slot of f_out is written by exactly one
// cell or ghost push, so the two halves may run at different times
int level_step_impl(ilbm_ctx *ctx, const ilbm_box *boxes, int nbox, const ilbm_level_params *p,
                    const int *mlo, const int *mhi, int part) {
  if (!ctx || !boxes || nbox <= 0 || part < 0 || part > 2 || (part && nbox != 1)) {
    set_error("level step: null argument");
    return ILBM_ERR_ARG;
  }
  int rc = check_params(ctx, p);
  if (rc) return rc;
  for (int n = 0; n < nbox; ++n)
    if (boxes[n].ngrow_f < 1) {
      set_error("f arrays need at least one ghost layer (edge cells push into it as scratch)");
      return ILBM_ERR_ARG;
    }
  if (p->ghost_mode == ILBM_GHOST_SELF) {
    if (nbox != 1) {
      set_error("self-fill ghost mode needs exactly one box covering the domain");
      return ILBM_ERR_ARG;
    }
    for (int d = 0; d < ctx->dim; ++d)
      if (boxes[0].lo[d] != p->domain_lo[d] || boxes[0].hi[d] != p->domain_hi[d]) {
        set_error("self-fill ghost mode: the box must equal the domain");
        return ILBM_ERR_ARG;
      }

  } else if (p->ghost_mode != ILBM_GHOST_CALLER) {
    set_error("unknown ghost mode");
    return ILBM_ERR_ARG;
  }
  for (int n = 0; n < nbox; ++n) {
    const ilbm_box &b = boxes[n];
    if ((rc = check_box(ctx, b, true))) return rc;
    if (p->ghost_mode == ILBM_GHOST_CALLER && b.ngrow_f < 1) {
      set_error("caller ghost mode needs ngrow_f >= 1");
      return ILBM_ERR_ARG;
    }
    if (p->ghost_mode == ILBM_GHOST_CALLER && (b.macro_in || b.force || b.force_prev) &&
        b.ngrow_m < 1) {
      set_error("caller ghost mode reads macro/force ghosts: needs ngrow_m >= 1");
      return ILBM_ERR_ARG;
    }
    if ((b.macro_in || b.macro_out || b.force || b.force_prev) &&
        (b.mstride[0] <= 0 || b.mstride[1] <= 0 || b.mstride[2] <= 0)) {
      set_error("box: macro/force strides must be positive");
      return ILBM_ERR_ARG;
    }
    if (b.f_in == b.f_out) {
      set_error("f_in and f_out must be distinct (two-lattice scheme)");
      return ILBM_ERR_ARG;
    }
  }
  // (the level's boxes are read in caller mode only)
  if (part == 0 && !mlo && p->ghost_mode == ILBM_GHOST_CALLER && (nbox > 1 || p->nlevel_boxes > 1))
    return level_step_boxes(ctx, boxes, nbox, p);
  for (int n = 0; n < nbox; ++n) {
    const ilbm_box &b = boxes[n];
    StepArgs a;
    if ((rc = fill_args(ctx, b, p, a))) return rc;
    if (mlo && mhi) {
      a.use_mbox = 1;
      for (int d = 0; d < 3; ++d) {
        a.mblo[d] = (d < ctx->dim) ? mlo[d] : 0;
        a.mbhi[d] = (d < ctx->dim) ? mhi[d] : 0;
      }
    }
    if (part == 0) {
      rc = ILBM_DISPATCH(ctx, launch_step, ctx, a);
    } else if (a.hi[ctx->dim - 1] == a.lo[ctx->dim - 1]) {
      // one cell along the split dimension: the first part takes it all
      if (part == 1) rc = ILBM_DISPATCH(ctx, launch_step_part, ctx, a, true);
    } else {
      const int e = ctx->dim - 1;  // split along the last dimension
      const int mid = a.lo[e] + (a.hi[e] - a.lo[e] + 1) / 2 - 1;
      if (part == 1)
        a.rhi[e] = mid;
      else
        a.rlo[e] = mid + 1;
      rc = ILBM_DISPATCH(ctx, launch_step_part, ctx, a, part == 1);
    }
    if (rc) return rc;
    if (part == 1) continue;  // macro_out once both halves have run
    if (b.macro_out) {
      StepArgs am = a;
      am.f_in = b.f_out;
      int rlo[3] = {a.lo[0], a.lo[1], a.lo[2]}, rhi[3] = {a.hi[0], a.hi[1], a.hi[2]};
      if (a.use_mbox)  // stored values are kept on the macro box only
        for (int d = 0; d < ctx->dim; ++d) {
          rlo[d] = std::max(rlo[d], a.mblo[d]);
          rhi[d] = std::min(rhi[d], a.mbhi[d]);
        }
      rc = ILBM_DISPATCH(ctx, launch_macro, ctx, am, rlo, rhi, b.macro_out);
      if (rc) return rc;
    }
  }
  return ILBM_OK;
}

}  // namespace ilbm

using namespace ilbm;

void *ilbm_ctx_scratch(ilbm_ctx *ctx, size_t n) {
  if (ctx->scratch_bytes >= n) return ctx->scratch;
  if (ctx->scratch) cudaFree(ctx->scratch);
  ctx->scratch = nullptr;
  ctx->scratch_bytes = 0;
  if (cudaMalloc(&ctx->scratch, n) != cudaSuccess) return nullptr;
  ctx->scratch_bytes = n;
  return ctx->scratch;
}

cudaError_t ilbm_ctx_malloc(ilbm_ctx *ctx, void **p, size_t bytes) {
  return cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 1), ctx->pool, ctx->stream);
}

void ilbm_ctx_free(ilbm_ctx *ctx, void *p) {
  if (p) cudaFreeAsync(p, ctx->stream);
}

extern "C" {

const char *ilbm_last_error(void) { return ilbm::get_error(); }

int ilbm_create(const ilbm_lattice *lat, int storage, int device, void *cuda_stream,
                ilbm_ctx **out) {
  if (!lat || !out) {
    set_error("ilbm_create: null argument");
    return ILBM_ERR_ARG;
  }
  *out = nullptr;
  if (storage < ILBM_STORAGE_F64 || storage > ILBM_STORAGE_F16_SCALED) {
    set_error("ilbm_create: unknown storage form");
    return ILBM_ERR_ARG;
  }
  // the lattice must be one of the three deck orderings, with w = wis/wim
  int dim = 0;
  auto match = [&](auto L) -> bool {
    using LL = decltype(L);
    if (lat->q != LL::Q) return false;
    for (int q = 0; q < LL::Q; ++q) {
      if (lat->cx[q] != double(LL::cx(q)) || lat->cy[q] != double(LL::cy(q)) ||
          lat->cz[q] != double(LL::cz(q)))
        return false;
      if (lat->wim[q] == 0.0 || lat->wis[q] / lat->wim[q] != LL::w(q)) return false;
    }
    dim = LL::D;
    return true;
  };
  if (!(match(Lat<9>{}) || match(Lat<19>{}) || match(Lat<27>{}))) {
    set_error("ilbm_create: lattice must be D2Q9, D3Q19 or D3Q27 in the reference deck order");
    return ILBM_ERR_UNSUPPORTED;
  }
  if (lat->dim != 0 && lat->dim != dim) {
    set_error("ilbm_create: lattice dimension mismatch");
    return ILBM_ERR_ARG;
  }
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
  auto *c = new ilbm_ctx();
  c->q = lat->q;
  for (int q = 0; q < lat->q; ++q) c->w[q] = lat->wis[q] / lat->wim[q];
  c->dim = dim;
  c->storage = storage;
  c->device = device;
  if (cuda_stream) {
    c->stream = static_cast<cudaStream_t>(cuda_stream);
  } else {
    e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      delete c;
      return cuda_fail(e, "cudaStreamCreate");
    }
    c->own_stream = true;
  }
  for (int s = 0; s < 16; ++s) {
    e = cudaEventCreate(&c->ev[s]);
    if (e != cudaSuccess) {
      ilbm_destroy(c);
      return cuda_fail(e, "cudaEventCreate");
    }
  }
  {
    // high-priority side stream for the immersed-boundary chain, which then
    // overlaps the collide-stream of the cells outside its band
    int lo_pri = 0, hi_pri = 0;
    cudaDeviceGetStreamPriorityRange(&lo_pri, &hi_pri);
    e = cudaStreamCreateWithPriority(&c->side, cudaStreamNonBlocking, hi_pri);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_join, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_rec, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      ilbm_destroy(c);
      return cuda_fail(e, "side stream");
    }
  }
  e = cudaMallocHost(&c->host_pinned, 64 * sizeof(double));
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) {
    cudaMemPoolProps pp = {};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = device;
    e = cudaMemPoolCreate(&c->pool, &pp);
    uint64_t keep = UINT64_MAX;  // never trim at synchronisation points
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  if (e != cudaSuccess) {
    ilbm_destroy(c);
    return cuda_fail(e, "ilbm_create");
  }
  *out = c;
  return ILBM_OK;
}

int ilbm_destroy(ilbm_ctx *ctx) {
  if (!ctx) return ILBM_OK;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  for (int s = 0; s < 16; ++s)
    if (ctx->ev[s]) cudaEventDestroy(ctx->ev[s]);
  for (int s = 0; s < ctx->nxev; ++s)
    if (ctx->xev[s]) cudaEventDestroy(ctx->xev[s]);
  delete[] ctx->xev;
  if (ctx->scratch) cudaFree(ctx->scratch);
  if (ctx->host_pinned) cudaFreeHost(ctx->host_pinned);
  if (ctx->side) {
    cudaStreamSynchronize(ctx->side);
    cudaStreamDestroy(ctx->side);
  }
  if (ctx->ev_fork) cudaEventDestroy(ctx->ev_fork);
  if (ctx->ev_join) cudaEventDestroy(ctx->ev_join);
  if (ctx->ev_done) cudaEventDestroy(ctx->ev_done);
  if (ctx->ev_rec) cudaEventDestroy(ctx->ev_rec);
  // a pool with allocations outstanding is released once they are freed
  if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
  if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
  return ILBM_OK;
}

int ilbm_sync(ilbm_ctx *ctx) {
  if (!ctx) return ILBM_ERR_ARG;
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_fail(e, "stream synchronize");
  return ILBM_OK;
}

void *ilbm_stream(ilbm_ctx *ctx) { return ctx ? (void *)ctx->stream : nullptr; }

}  // extern "C"

// a recorded sequence of the context's launches, instantiated once
struct ilbm_graph {
  cudaGraphExec_t exec = nullptr;
  int64_t kernels = 0;  // kernel nodes: what one replay adds to the launch count
};

extern "C" {

int ilbm_graph_begin(ilbm_ctx *ctx) {
  if (!ctx) return ILBM_ERR_ARG;
  if (ctx->capture_launch0 >= 0) {
    set_error("ilbm_graph_begin: a capture is already open on this context");
    return ILBM_ERR_ARG;
  }
  cudaSetDevice(ctx->device);
  // thread-local: launches other host threads make meanwhile are not recorded
  cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cuda_fail(e, "ilbm_graph_begin");
  ctx->capture_launch0 = ctx->launches;
  return ILBM_OK;
}

int ilbm_graph_end(ilbm_ctx *ctx, ilbm_graph **out) {
  if (!ctx || !out) return ILBM_ERR_ARG;
  *out = nullptr;
  if (ctx->capture_launch0 < 0) {
    set_error("ilbm_graph_end: no capture open on this context");
    return ILBM_ERR_ARG;
  }
  ctx->launches = ctx->capture_launch0;  // the recorded launches did not run
  ctx->capture_launch0 = -1;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
  if (e != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    return cuda_fail(e != cudaSuccess ? e : cudaErrorStreamCaptureInvalidated, "ilbm_graph_end");
  }
  size_t nn = 0;
  e = cudaGraphGetNodes(g, nullptr, &nn);
  std::vector<cudaGraphNode_t> nodes(nn);
  if (e == cudaSuccess && nn) e = cudaGraphGetNodes(g, nodes.data(), &nn);
  int64_t kernels = 0;
  for (size_t i = 0; e == cudaSuccess && i < nn; ++i) {
    cudaGraphNodeType t;
    e = cudaGraphNodeGetType(nodes[i], &t);
    if (e == cudaSuccess && t == cudaGraphNodeTypeKernel) ++kernels;
  }
  cudaGraphExec_t exec = nullptr;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return cuda_fail(e, "ilbm_graph_end: instantiate");
  ilbm_graph *h = new ilbm_graph;
  h->exec = exec;
  h->kernels = kernels;
  *out = h;
  return ILBM_OK;
}

int ilbm_graph_launch(ilbm_ctx *ctx, const ilbm_graph *g) {
  if (!ctx || !g || !g->exec) return ILBM_ERR_ARG;
  cudaError_t e = cudaGraphLaunch(g->exec, ctx->stream);
  if (e != cudaSuccess) return cuda_fail(e, "ilbm_graph_launch");
  ctx->launches += g->kernels;
  return ILBM_OK;
}

int ilbm_graph_destroy(ilbm_graph *g) {
  if (!g) return ILBM_OK;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  delete g;
  return ILBM_OK;
}

static cudaEvent_t *event_slot(ilbm_ctx *ctx, int slot) {
  if (slot < 0 || slot >= 16 + 8192) return nullptr;
  if (slot < 16) return &ctx->ev[slot];
  const int x = slot - 16;
  if (x >= ctx->nxev) {
    const int n = std::max(x + 1, std::max(64, 2 * ctx->nxev));
    auto *nv = new cudaEvent_t[n];
    for (int i = 0; i < ctx->nxev; ++i) nv[i] = ctx->xev[i];
    for (int i = ctx->nxev; i < n; ++i) nv[i] = nullptr;
    delete[] ctx->xev;
    ctx->xev = nv;
    ctx->nxev = n;
  }
  if (!ctx->xev[x] && cudaEventCreate(&ctx->xev[x]) != cudaSuccess) return nullptr;
  return &ctx->xev[x];
}

int ilbm_event_record(ilbm_ctx *ctx, int slot) {
  if (!ctx) return ILBM_ERR_ARG;
  cudaEvent_t *ev = event_slot(ctx, slot);
  if (!ev) {
    set_error("event slot out of range (0..8207)");
    return ILBM_ERR_ARG;
  }
  cudaError_t e = cudaEventRecord(*ev, ctx->stream);
  if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord");
  return ILBM_OK;
}

int ilbm_event_elapsed_ms(ilbm_ctx *ctx, int a, int b, float *ms) {
  if (!ctx || !ms) return ILBM_ERR_ARG;
  cudaEvent_t *ea = event_slot(ctx, a), *eb = event_slot(ctx, b);
  if (!ea || !eb) {
    set_error("event slot out of range");
    return ILBM_ERR_ARG;
  }
  cudaError_t e = cudaEventSynchronize(*eb);
  if (e != cudaSuccess) return cuda_fail(e, "cudaEventSynchronize");
  e = cudaEventElapsedTime(ms, *ea, *eb);
  if (e != cudaSuccess) return cuda_fail(e, "cudaEventElapsedTime");
  return ILBM_OK;
}

int64_t ilbm_kernel_launches(const ilbm_ctx *ctx) { return ctx ? ctx->launches : -1; }

int ilbm_storage_bytes(const ilbm_ctx *ctx, int *sb, int *rb) {
  if (!ctx) return ILBM_ERR_ARG;
  const int s = ctx->storage == ILBM_STORAGE_F64 ? 8 : (ctx->storage == ILBM_STORAGE_F32_SHIFT ? 4 : 2);
  if (sb) *sb = s;
  if (rb) *rb = ctx->storage == ILBM_STORAGE_F64 ? 8 : 4;
  return ILBM_OK;
}

int ilbm_level_step(ilbm_ctx *ctx, const ilbm_box *boxes, int nbox, const ilbm_level_params *p) {
  return level_step_impl(ctx, boxes, nbox, p, nullptr, nullptr, 0);
}

int ilbm_compute_macro(ilbm_ctx *ctx, const ilbm_box *box, const ilbm_level_params *p,
                       const void *f, const void *force, void *macro_out, const int lo[3],
                       const int hi[3]) {
  if (!ctx || !box || !f || !macro_out) {
    set_error("ilbm_compute_macro: null argument");
    return ILBM_ERR_ARG;
  }
  StepArgs a;
  int rc = fill_args(ctx, *box, p, a);
  if (rc) return rc;
  a.f_in = f;
  a.force = force;
  if (!p) {
    for (int d = 0; d < 3; ++d) {
      a.flo[d] = -(1 << 30);
      a.fhi[d] = (1 << 30);
    }
  }
  int rlo[3], rhi[3];
  for (int d = 0; d < 3; ++d) {
    const bool use = d < ctx->dim;
    rlo[d] = use ? std::max(lo ? lo[d] : box->lo[d], box->lo[d]) : 0;
    rhi[d] = use ? std::min(hi ? hi[d] : box->hi[d], box->hi[d]) : 0;
  }
  return ILBM_DISPATCH(ctx, launch_macro, ctx, a, rlo, rhi, macro_out);
}

int ilbm_init_equilibrium(ilbm_ctx *ctx, const ilbm_box *box) {
  if (!ctx || !box || !box->f_in || !box->f_out || !box->macro_in) {
    set_error("ilbm_init_equilibrium: f_in, f_out and macro_in are required");
    return ILBM_ERR_ARG;
  }
  if (box->ngrow_m < box->ngrow_f) {
    set_error("ilbm_init_equilibrium: macro ghost width must cover the f ghost width");
    return ILBM_ERR_ARG;
  }
  StepArgs a;
  int rc = fill_args(ctx, *box, nullptr, a);
  if (rc) return rc;
  return ILBM_DISPATCH(ctx, launch_init, ctx, a, box->ngrow_f);
}


int ilbm_derived_fields(ilbm_ctx *ctx, const ilbm_box *box, const ilbm_level_params *p,
                        const void *f, const void *force_prev, const double dx[3], void *vor,
                        void *pres, double *vort_max) {
  if (!ctx || !box || !p || !f || !dx) {
    set_error("ilbm_derived_fields: null argument");
    return ILBM_ERR_ARG;
  }
  int rc = check_params(ctx, p);
  if (rc) return rc;
  if (p->ghost_mode != ILBM_GHOST_SELF) {
    set_error("ilbm_derived_fields: needs self-filled ghosts (one box equal to the domain)");
    return ILBM_ERR_UNSUPPORTED;
  }
  for (int d = 0; d < ctx->dim; ++d)
    if (box->lo[d] != p->domain_lo[d] || box->hi[d] != p->domain_hi[d]) {
      set_error("ilbm_derived_fields: the box must equal the domain");
      return ILBM_ERR_ARG;
    }
  if ((vor || pres) && (box->mstride[0] <= 0 || box->mstride[1] <= 0)) {
    set_error("ilbm_derived_fields: macro strides must be positive");
    return ILBM_ERR_ARG;
  }
  ilbm_box b = *box;
  b.f_in = const_cast<void *>(f);
  b.f_out = nullptr;
  b.macro_in = nullptr;
  b.force_prev = const_cast<void *>(force_prev);
  DeriveArgs d;
  std::memset(&d, 0, sizeof(d));
  d.dim = ctx->dim;
  int64_t nb = 1, ncell = 1;
  int blo[3] = {0, 0, 0}, bn[3] = {1, 1, 1};
  for (int q = 0; q < 3; ++q) {
    d.lo[q] = (q < ctx->dim) ? box->lo[q] : 0;
    d.hi[q] = (q < ctx->dim) ? box->hi[q] : 0;
    d.mgl[q] = (q < ctx->dim) ? box->lo[q] - box->ngrow_m : 0;
    if (q < ctx->dim) {
      blo[q] = box->lo[q] - 1;
      bn[q] = box->hi[q] - box->lo[q] + 3;
    }
    d.blo[q] = blo[q];
    d.bn[q] = bn[q];
    nb *= bn[q];
    ncell *= (d.hi[q] - d.lo[q] + 1);
  }
  d.nb = nb;
  d.ms0 = box->mstride[0];
  d.ms1 = box->mstride[1];
  for (int q = 0; q < 3; ++q) d.dx[q] = dx[q];  // the level's xCellSize, yCellSize, zCellSize
  const int blocks = (int)std::min<int64_t>((ncell + 255) / 256, 1184);
  double *scr = static_cast<double *>(ilbm_ctx_scratch(ctx, (4 * nb + blocks + 8) * sizeof(double)));
  if (!scr) {
    set_error("ilbm_derived_fields: scratch allocation failed");
    return ILBM_ERR_NOMEM;
  }
  double *EV = scr, *RHO = scr + 3 * nb, *bmax = scr + 4 * nb, *out = bmax + blocks;
  if ((rc = band_macro(ctx, b, p, blo, bn, EV, RHO, ctx->stream))) return rc;
  if (ctx->storage == ILBM_STORAGE_F64)
    k_derive<double><<<blocks, 256, 0, ctx->stream>>>(d, EV, RHO, static_cast<double *>(vor),
                                                      static_cast<double *>(pres), bmax);
  else
    k_derive<float><<<blocks, 256, 0, ctx->stream>>>(d, EV, RHO, static_cast<float *>(vor),
                                                     static_cast<float *>(pres), bmax);
  k_max_final<<<1, 32, 0, ctx->stream>>>(bmax, blocks, out);
  ctx->launches += 2;
  double mx = 0.0;
  cudaMemcpyAsync(&mx, out, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_fail(e, "ilbm_derived_fields");
  if (vort_max) *vort_max = mx;
  return ILBM_OK;
}

int ilbm_tag_cells(ilbm_ctx *ctx, const ilbm_box *box, const void *vor, double threshold,
                   int use_box, const double box_lo[3], const double box_hi[3],
                   double no_refine_xlo, double no_refine_xhi, const double prob_lo[3],
                   const double prob_hi[3], const double dx[3], const double *levelset,
                   void *tags, int64_t *ntagged) {
  if (!ctx || !box || !vor || !tags || !prob_lo || !prob_hi || !dx || (use_box && (!box_lo || !box_hi))) {
    set_error("ilbm_tag_cells: null argument");
    return ILBM_ERR_ARG;
  }
  TagArgs g;
  std::memset(&g, 0, sizeof(g));
  g.dim = ctx->dim;
  int64_t ncell = 1;
  for (int q = 0; q < 3; ++q) {
    g.lo[q] = (q < ctx->dim) ? box->lo[q] : 0;
    g.hi[q] = (q < ctx->dim) ? box->hi[q] : 0;
    g.mgl[q] = (q < ctx->dim) ? box->lo[q] - box->ngrow_m : 0;
    ncell *= (g.hi[q] - g.lo[q] + 1);
    g.plo[q] = prob_lo[q];
    g.phi[q] = prob_hi[q];
    g.dx[q] = dx[q];
    if (use_box) {
      g.box_lo[q] = box_lo[q];
      g.box_hi[q] = box_hi[q];
    }
  }
  g.ms0 = box->mstride[0];
  g.ms1 = box->mstride[1];
  g.threshold = threshold;
  g.use_box = use_box;
  g.nr_lo = no_refine_xlo;
  g.nr_hi = no_refine_xhi;
  if (levelset) {
    if (!(levelset[4] >= 0.0) || !(levelset[5] > 0.0)) {
      set_error("ilbm_tag_cells: level-set band cells must be >= 0 and dx_min > 0");
      return ILBM_ERR_ARG;
    }
    g.use_ls = 1;
    for (int q = 0; q < 3; ++q) g.ls_c[q] = levelset[q];
    g.ls_r = levelset[3];
    // (n_cells_band + 0.5) * dx_min
    g.ls_band = (std::floor(levelset[4]) + 0.5) * levelset[5];
  }
  unsigned long long *cnt =
      static_cast<unsigned long long *>(ilbm_ctx_scratch(ctx, 8 * sizeof(unsigned long long)));
  if (!cnt) {
    set_error("ilbm_tag_cells: scratch allocation failed");
    return ILBM_ERR_NOMEM;
  }
  cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), ctx->stream);
  const int blocks = (int)std::min<int64_t>((ncell + 255) / 256, 1184);
  if (ctx->storage == ILBM_STORAGE_F64)
    k_tags<double><<<blocks, 256, 0, ctx->stream>>>(g, static_cast<const double *>(vor),
                                                    static_cast<unsigned char *>(tags), cnt);
  else
    k_tags<float><<<blocks, 256, 0, ctx->stream>>>(g, static_cast<const float *>(vor),
                                                   static_cast<unsigned char *>(tags), cnt);
  ctx->launches++;
  unsigned long long h = 0;
  cudaMemcpyAsync(&h, cnt, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream);
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_fail(e, "ilbm_tag_cells");
  if (ntagged) *ntagged = (int64_t)h;
  return ILBM_OK;
}

}  // extern "C"
