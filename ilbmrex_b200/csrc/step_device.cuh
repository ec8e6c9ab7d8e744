// Device helpers of the level step shared by its kernels (level_step.cuh) and
// the macro, initialisation and band kernels (lbm_step.cu): cell indices,
// population and force loads, the ghost rules of a self-filled level.
#pragma once

#include "ilbm_common.cuh"
#include "step_args.cuh"

namespace ilbm {

__device__ __forceinline__ int64_t fidx(const StepArgs &a, int i, int j, int k) {
  return (int64_t)(i - a.fgl[0]) + (int64_t)(j - a.fgl[1]) * a.fs0 +
         (int64_t)(k - a.fgl[2]) * a.fs1;
}
__device__ __forceinline__ int64_t midx(const StepArgs &a, int i, int j, int k) {
  return (int64_t)(i - a.mgl[0]) + (int64_t)(j - a.mgl[1]) * a.ms0 +
         (int64_t)(k - a.mgl[2]) * a.ms1;
}

template <class L>
__device__ __forceinline__ bool in_domain(const StepArgs &a, int i, int j, int k) {
  if (i < a.dlo[0] || i > a.dhi[0] || j < a.dlo[1] || j > a.dhi[1]) return false;
  if (L::D == 3 && (k < a.dlo[2] || k > a.dhi[2])) return false;
  return true;
}

// per-direction storage factor for the F16 form: w_q / scale
template <class L, int S>
__device__ __forceinline__ float sfac(const StepArgs &a, int q) {
  if (S == ILBM_STORAGE_F16_SCALED) return float(L::w(q)) / a.f16_scale;
  return 1.0f;
}

template <class L, int S>
__device__ __forceinline__ typename Store<S>::R ldf(const StepArgs &a, int64_t base, int q) {
  using T = typename Store<S>::T;
  return Store<S>::load(static_cast<const T *>(a.f_in) + base + q * a.fs2, sfac<L, S>(a, q));
}

template <class R>
__device__ __forceinline__ R ldm(const void *p, int64_t idx) {
  return static_cast<const R *>(p)[idx];
}

// force at a cell (F^n or F^{n-1}); zero outside the force region
template <class L, class R>
__device__ __forceinline__ void load_force(const StepArgs &a, const void *F, int i, int j,
                                           int k, R &fx, R &fy, R &fz) {
  if (F == nullptr) {
    if (a.use_uniform) {
      fx = R(a.uf[0]);
      fy = R(a.uf[1]);
      fz = R(a.uf[2]);
    } else {
      fx = fy = fz = R(0);
    }
    return;
  }
  if (i < a.flo[0] || i > a.fhi[0] || j < a.flo[1] || j > a.fhi[1] ||
      (L::D == 3 && (k < a.flo[2] || k > a.fhi[2]))) {
    fx = fy = fz = R(0);
    return;
  }
  const int64_t m = midx(a, i, j, k);
  fx = ldm<R>(F, m);
  fy = ldm<R>(F, m + a.ms2);
  fz = (L::D == 3) ? ldm<R>(F, m + 2 * a.ms2) : R(0);
}

// ---------------------------------------------------------------------------
// Ghost synthesis (pre-collision values of physical-boundary ghosts), with the
// FillPatch semantics the reference relies on: periodic images first, then per
// ghost cell AMReX's foextrap fill followed by mesoscopicBcFill
// (Source/BC/bc_fill.H:303-347: user_2 face mirror > user_1 copy > ext_dir
// non-equilibrium extrapolation, mirror = nearest domain cell).
// ---------------------------------------------------------------------------
template <class L>
__device__ __forceinline__ bool first_face(const StepArgs &a, const int *g, int type, int &bd,
                                           int &lo_side) {
#pragma unroll
  for (int d = 0; d < L::D; ++d) {
    if (g[d] < a.dlo[d] && a.bclo[d] == type) { bd = d; lo_side = 1; return true; }
    if (g[d] > a.dhi[d] && a.bchi[d] == type) { bd = d; lo_side = 0; return true; }
  }
  return false;
}

// Resolve a ghost cell to either a source cell in the domain (copy) or a
// boundary formula on a mirror cell.  kind: 0 copy src, 1 user_1 copy of
// mirror, 2 ext_dir NEQ, 3 user_2 face-mirror NEQ.
template <class L>
__device__ __forceinline__ int ghost_rule(const StepArgs &a, const int *g, int *src, int &bd,
                                          int &lo_side) {
  int cur[3] = {g[0], g[1], g[2]};
  for (int it = 0; it < 4; ++it) {
    bool inside = true, wrappable = true;
#pragma unroll
    for (int d = 0; d < L::D; ++d) {
      const bool out = cur[d] < a.dlo[d] || cur[d] > a.dhi[d];
      if (out) {
        inside = false;
        if (!a.periodic[d]) wrappable = false;
      }
    }
    if (inside || wrappable) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        int c = cur[d];
        if (d < L::D && a.periodic[d]) {
          const int n = a.dhi[d] - a.dlo[d] + 1;
          while (c < a.dlo[d]) c += n;  // a ghost lies a cell or two outside
          while (c > a.dhi[d]) c -= n;
        }
        src[d] = c;
      }
      return 0;
    }
    if (it == 0) {
      int m[3] = {cur[0], cur[1], cur[2]};
#pragma unroll
      for (int d = 0; d < L::D; ++d) m[d] = min(max(cur[d], a.dlo[d]), a.dhi[d]);
      if (first_face<L>(a, cur, ILBM_BC_USER_2, bd, lo_side)) { src[0] = m[0]; src[1] = m[1]; src[2] = m[2]; return 3; }
      if (first_face<L>(a, cur, ILBM_BC_USER_1, bd, lo_side)) { src[0] = m[0]; src[1] = m[1]; src[2] = m[2]; return 1; }
      if (first_face<L>(a, cur, ILBM_BC_EXT_DIR, bd, lo_side)) { src[0] = m[0]; src[1] = m[1]; src[2] = m[2]; return 2; }
    }
    // foextrap: the last dimension with a foextrap face wins (FilccCell order)
    int dsel = -1;
#pragma unroll
    for (int d = 0; d < L::D; ++d) {
      if (cur[d] < a.dlo[d] && a.bclo[d] == ILBM_BC_FOEXTRAP) dsel = d;
      else if (cur[d] > a.dhi[d] && a.bchi[d] == ILBM_BC_FOEXTRAP) dsel = d;
    }
    if (dsel < 0) break;
#pragma unroll
    for (int d = 0; d < L::D; ++d)  // (constant subscripts: cur stays in registers)
      if (d == dsel) cur[d] = (cur[d] < a.dlo[d]) ? a.dlo[d] : a.dhi[d];
  }
  src[0] = min(max(g[0], a.dlo[0]), a.dhi[0]);
  src[1] = min(max(g[1], a.dlo[1]), a.dhi[1]);
  src[2] = (L::D == 3) ? min(max(g[2], a.dlo[2]), a.dhi[2]) : 0;
  return 0;
}

}  // namespace ilbm
