// Device helpers of the level step shared by its kernels (level_step.cuh) and
// the macro, initialisation and band kernels (lbm_step.cu): cell indices,
// population and force loads, the ghost rules of a self-filled level, rho and u
// of a cell of the immersed boundary's band.
#pragma once

#include "ilbm_common.cuh"
#include "step_args.cuh"

namespace ilbm {

// n / d by a multiplication (n < 2^31): d's magic from the host (div_magic)
__device__ __forceinline__ uint32_t fast_div(uint32_t n, const DivMagic &d) {
  return (__umulhi(n, d.mul) + n) >> d.shift;
}

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

// ---------------------------------------------------------------------------
// Band macro for the immersed boundary: rho, u, v, w (FP64) on the cells of
// the IB support band, including up to two ghost layers outside the domain.
// Valid cells: from macro_in, or from f^n and F^{n-1} (the value the
// reference's macro pass stored).  Ghost cells: FillPatchMacro semantics
// (periodic image, foextrap, macroBcFill: user_2 mirrored state, user_1 /
// ext_dir prescribed state; Source/BC/bc_fill.H:69-142, 263-301).
// ---------------------------------------------------------------------------
template <class L, int S>
__device__ void macro_at(const StepArgs &a, int i, int j, int k, double *m4) {
  if (stored_macro_at(a, i, j, k)) {
    const int64_t m = midx(a, i, j, k);
    if (S == ILBM_STORAGE_F64) {
      m4[0] = ldm<double>(a.macro_in, m);
      m4[1] = ldm<double>(a.macro_in, m + a.ms2);
      m4[2] = ldm<double>(a.macro_in, m + 2 * a.ms2);
      m4[3] = (L::D == 3) ? ldm<double>(a.macro_in, m + 3 * a.ms2) : 0.0;
    } else {
      m4[0] = ldm<float>(a.macro_in, m);
      m4[1] = ldm<float>(a.macro_in, m + a.ms2);
      m4[2] = ldm<float>(a.macro_in, m + 2 * a.ms2);
      m4[3] = (L::D == 3) ? ldm<float>(a.macro_in, m + 3 * a.ms2) : 0.0;
    }
    return;
  }
  const int64_t b = fidx(a, i, j, k);
  if (S == ILBM_STORAGE_F64) {
    double f[L::Q];
#pragma unroll
    for (int q = 0; q < L::Q; ++q) f[q] = ldf<L, S>(a, b, q);
    double px, py, pz;
    load_force<L, double>(a, a.force_prev, i, j, k, px, py, pz);
    moments64<L>(f, px, py, pz, m4[0], m4[1], m4[2], m4[3]);
    if (L::D != 3) m4[3] = 0.0;
  } else {
    float g[L::Q];
#pragma unroll
    for (int q = 0; q < L::Q; ++q) g[q] = ldf<L, S>(a, b, q);
    float px, py, pz, drho, u, v, w;
    load_force<L, float>(a, a.force_prev, i, j, k, px, py, pz);
    moments32<L>(g, px, py, pz, drho, u, v, w);
    m4[0] = 1.0 + double(drho);
    m4[1] = u;
    m4[2] = v;
    m4[3] = (L::D == 3) ? double(w) : 0.0;
  }
}

// rho, u, v, w of one band cell
template <class L, int S>
__device__ __forceinline__ void band_macro_value(const StepArgs &a, int i, int j, int k, double *m4) {
  const int g[3] = {i, j, k};
  const bool in = in_domain<L>(a, g[0], g[1], g[2]);
  if (in || (a.macro_in && !a.self_fill)) {
    // caller-filled macros carry their own ghost values
    macro_at<L, S>(a, g[0], g[1], L::D == 3 ? g[2] : 0, m4);
    return;
  }
  int src[3], bd = 0, lo_side = 1;
  const int kind = ghost_rule<L>(a, g, src, bd, lo_side);
  macro_at<L, S>(a, src[0], src[1], L::D == 3 ? src[2] : 0, m4);
  const double *bv = lo_side ? a.bvlo[bd] : a.bvhi[bd];
  if (kind == 3) {
    m4[0] = fmax(1.0e-20, X::sub(X::mul(2.0, bv[0]), m4[0]));
    m4[1] = X::sub(X::mul(2.0, bv[1]), m4[1]);
    m4[2] = X::sub(X::mul(2.0, bv[2]), m4[2]);
    m4[3] = X::sub(X::mul(2.0, bv[3]), m4[3]);
  } else if (kind == 1 || kind == 2) {
    m4[0] = bv[0];
    m4[1] = bv[1];
    m4[2] = bv[2];
    m4[3] = bv[3];
  }
}

template <class L, int S>
__device__ __forceinline__ void band_macro_cell(const StepArgs &a, int blo0, int blo1, int blo2,
                                                int bn0, int bn1, int64_t nb, int64_t t,
                                                double *EV, double *RHO) {
  double m4[4];
  band_macro_value<L, S>(a, blo0 + (int)(t % bn0), blo1 + (int)((t / bn0) % bn1),
                         blo2 + (int)(t / ((int64_t)bn0 * bn1)), m4);
  EV[t] = m4[1];
  EV[t + nb] = m4[2];
  EV[t + 2 * nb] = (L::D == 3) ? m4[3] : 0.0;
  RHO[t] = m4[0];
}

}  // namespace ilbm
