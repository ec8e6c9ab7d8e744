// The level-step kernels (collide + push, with the ghost shell's push) and
// their launches, included by the translation units that instantiate them
// (step_q*.cu).
#pragma once

#include <algorithm>

#include "step_device.cuh"
#include "step_launch.h"

namespace ilbm {

// Populations that enter the box from its layer-1 ghost shell are pushed here,
// one thread per ghost cell: the pre-collision boundary value (self-fill: the
// FillPatch rules above on f^n of the domain; caller-filled: the ghost value
// as given), or, for a ghost covered by another box of the level, that cell's
// post-collision value.  Ghosts that are periodic images (self-fill) and
// halfway bounce-back ghosts are left to the owning cells' push.  A ghost cell
// is owned by the slab of its lowest dimension outside the box (periodic
// dimensions excluded in self-fill mode, whose slabs do not exist), so the
// shell is one sequence of cells: slab d holds the cells outside the box in
// dimension d, inside it in the active dimensions below d, and on the grown
// range of the others (StepArgs::goff, filled by ghost_offsets).
// The work runs in blocks spread among those of the k_step launch (it writes only
// slots that no cell's push writes, and reads only f^n), so its strided
// accesses overlap the main stream instead of preceding it.  It is bound by
// latency: one thread's chain is one ghost's index, its loads in flight
// together, and its stores.  A thread that walked the 2 D slabs one after
// another, each with 64-bit index divisions and a load per direction before
// its store, was the tail of every small launch: a 50 x 50 x 45 FP64 box with
// covered ghosts took 61 us against 5 us of traffic, and twelve of them 774 us
// against 320 us with one ghost per thread; the three-level 1024 x 512
// cylinder 213 -> 182 us per coarse step.  Loading only the entering
// directions of a copied ghost matters too: all 19 made the two-level sphere
// 1.3% slower than before instead of 1.3% faster.
template <class L>
__device__ __forceinline__ bool ghost_active(const StepArgs &a, int d) {
  return !(a.self_fill && a.periodic[d]);
}

template <class L, int S>
__device__ __noinline__ void ghost_push(const StepArgs &a, const int (*lb)[6], uint32_t gid, uint32_t gstride) {
  using T = typename Store<S>::T;
  using R = typename Store<S>::R;
  T *fo = static_cast<T *>(a.f_out);
  const uint32_t total = a.goff[3];
  for (uint32_t t = gid; t < total; t += gstride) {
    const int d = (int)(t >= a.goff[1]) + (int)(L::D == 3 && t >= a.goff[2]);
    uint32_t r = t - (d == 0 ? 0u : (d == 1 ? a.goff[1] : a.goff[2]));
    int g[3] = {0, 0, 0};
#pragma unroll
    for (int e = 0; e < L::D; ++e) {
      const bool inner = e < d && ghost_active<L>(a, e);
      const uint32_t n = (uint32_t)(a.hi[e] - a.lo[e] + 1);
      const uint32_t ext = (e == d) ? 2u : (inner ? n : n + 2u);
      const uint32_t c = (e == L::D - 1) ? r : r % ext;
      r /= ext;
      g[e] = (e == d) ? (c ? a.hi[e] + 1 : a.lo[e] - 1) : a.lo[e] + (int)c - (inner ? 0 : 1);
    }
    // classify the ghost against the domain
    bool phys = false, pure_u1 = true;
#pragma unroll
    for (int e = 0; e < L::D; ++e) {
      int sd = 0;
      if (g[e] < a.dlo[e]) sd = -1;
      else if (g[e] > a.dhi[e]) sd = 1;
      if (sd == 0) continue;
      if (a.periodic[e]) {
        pure_u1 = false;
      } else {
        phys = true;
        if ((sd < 0 ? a.bclo[e] : a.bchi[e]) != ILBM_BC_USER_1) pure_u1 = false;
      }
    }
    if (a.self_fill && !phys) continue;  // periodic image: the wrapping push delivers it
    if (phys && pure_u1) continue;       // halfway bounce-back: reflected by the cell
    const int gk = (L::D == 3) ? g[2] : 0;
    // source of the ghost's populations
    int mode;  // 0 copy from src (raw), 1 NEQ boundary formula on src, 2 collide the ghost
    int src[3] = {g[0], g[1], gk}, bd = 0, lo_side = 1, kind = 0;
    if (phys && a.self_fill) {
      kind = ghost_rule<L>(a, g, src, bd, lo_side);
      mode = (kind <= 1) ? 0 : 1;
    } else if (phys) {
      mode = 0;  // caller-filled physical ghost, as given
    } else {
      int gw[3] = {g[0], g[1], gk};
#pragma unroll
      for (int e = 0; e < L::D; ++e)
        if (a.periodic[e]) {
          const int nn = a.dhi[e] - a.dlo[e] + 1;
          while (gw[e] < a.dlo[e]) gw[e] += nn;
          while (gw[e] > a.dhi[e]) gw[e] -= nn;
        }
      bool covered = false;
      for (int b = 0; b < a.nlb && !covered; ++b)
        covered = gw[0] >= lb[b][0] && gw[0] <= lb[b][3] && gw[1] >= lb[b][1] &&
                  gw[1] <= lb[b][4] && (L::D == 2 || (gw[2] >= lb[b][2] && gw[2] <= lb[b][5]));
      mode = covered ? 2 : 0;  // not covered: coarse-fine ghost, as given
    }
    const int64_t sb = fidx(a, src[0], src[1], L::D == 3 ? src[2] : 0);
    // the directions that enter the box, and the loads the ghost needs (those
    // directions; all of them where moments are formed), in flight together
    bool into[3][3];
#pragma unroll
    for (int e = 0; e < 3; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int x = ((e == 2) ? gk : g[e]) + c - 1;
        into[e][c] = x >= a.lo[e] && x <= a.hi[e];
      }
    auto enters = [&](int q) {
      return into[0][L::cx(q) + 1] && into[1][L::cy(q) + 1] && into[2][L::cz(q) + 1];
    };
    R fs[L::Q];
#pragma unroll
    for (int q = 0; q < L::Q; ++q) fs[q] = (mode != 0 || enters(q)) ? ldf<L, S>(a, sb, q) : R(0);
    // per-ghost state for the NEQ formula / the collision
    double r64 = 0, u64 = 0, v64 = 0, w64 = 0, rt64 = 0, ut64 = 0, vt64 = 0, wt64 = 0;
    float dr32 = 0, u32 = 0, v32 = 0, w32 = 0, drt32 = 0, ut32 = 0, vt32 = 0, wt32 = 0;
    R gFx = R(0), gFy = R(0), gFz = R(0);
    bool ghf = false;
    if (mode == 1) {
      // applyExtDirMesoscopic / applyFaceMirroredMesoscopic, bc_fill.H:159-261
      const double *bv = lo_side ? a.bvlo[bd] : a.bvhi[bd];
      if (S == ILBM_STORAGE_F64) {
        double rhonp = 0.0, unp = 0.0, vnp = 0.0, wnp = 0.0;
#pragma unroll
        for (int p = 0; p < L::Q; ++p) {
          const double fp = fs[p];
          rhonp = X::add(rhonp, fp);
          unp = X::add(unp, X::mul(double(L::cx(p)), fp));
          vnp = X::add(vnp, X::mul(double(L::cy(p)), fp));
          wnp = X::add(wnp, X::mul(double(L::cz(p)), fp));
        }
        rhonp = fmax(rhonp, 1.0e-20);
        r64 = rhonp;
        u64 = X::div(unp, rhonp);
        v64 = X::div(vnp, rhonp);
        w64 = X::div(wnp, rhonp);
        rt64 = bv[0]; ut64 = bv[1]; vt64 = bv[2]; wt64 = bv[3];
        if (kind == 3) {
          rt64 = fmax(1.0e-20, X::sub(X::mul(2.0, bv[0]), r64));
          ut64 = X::sub(X::mul(2.0, bv[1]), u64);
          vt64 = X::sub(X::mul(2.0, bv[2]), v64);
          wt64 = X::sub(X::mul(2.0, bv[3]), w64);
        }
      } else {
        float rr = 0.f, m1 = 0.f, m2 = 0.f, m3 = 0.f;
#pragma unroll
        for (int p = 0; p < L::Q; ++p) {
          const float gp = fs[p];
          rr += gp;
          if (L::cx(p)) m1 += float(L::cx(p)) * gp;
          if (L::cy(p)) m2 += float(L::cy(p)) * gp;
          if (L::cz(p)) m3 += float(L::cz(p)) * gp;
        }
        const float rho = fmaxf(1.0f + rr, 1.0e-20f);
        dr32 = rho - 1.0f;
        u32 = m1 / rho; v32 = m2 / rho; w32 = m3 / rho;
        drt32 = float(bv[0]) - 1.0f; ut32 = float(bv[1]); vt32 = float(bv[2]); wt32 = float(bv[3]);
        if (kind == 3) {
          drt32 = fmaxf(1.0e-20f, 2.0f * float(bv[0]) - rho) - 1.0f;
          ut32 = 2.0f * float(bv[1]) - u32;
          vt32 = 2.0f * float(bv[2]) - v32;
          wt32 = 2.0f * float(bv[3]) - w32;
        }
      }
    } else if (mode == 2) {
      load_force<L, R>(a, a.force, g[0], g[1], gk, gFx, gFy, gFz);
      ghf = !(gFx == R(0) && gFy == R(0) && gFz == R(0));
      if (stored_macro_at(a, g[0], g[1], gk)) {
        const int64_t m = midx(a, g[0], g[1], gk);
        if (S == ILBM_STORAGE_F64) {
          r64 = ldm<double>(a.macro_in, m);
          u64 = ldm<double>(a.macro_in, m + a.ms2);
          v64 = ldm<double>(a.macro_in, m + 2 * a.ms2);
          w64 = (L::D == 3) ? ldm<double>(a.macro_in, m + 3 * a.ms2) : 0.0;
        } else {
          dr32 = ldm<float>(a.macro_in, m) - 1.0f;
          u32 = ldm<float>(a.macro_in, m + a.ms2);
          v32 = ldm<float>(a.macro_in, m + 2 * a.ms2);
          w32 = (L::D == 3) ? ldm<float>(a.macro_in, m + 3 * a.ms2) : 0.0f;
        }
      } else if (S == ILBM_STORAGE_F64) {
        double px, py, pz;
        load_force<L, double>(a, a.force_prev, g[0], g[1], gk, px, py, pz);
        moments64<L>(reinterpret_cast<const double *>(fs), px, py, pz, r64, u64, v64, w64);
        if (L::D != 3) w64 = 0.0;
      } else {
        float px, py, pz;
        load_force<L, float>(a, a.force_prev, g[0], g[1], gk, px, py, pz);
        moments32<L>(reinterpret_cast<const float *>(fs), px, py, pz, dr32, u32, v32, w32);
      }
    }
#pragma unroll
    for (int q = 1; q < L::Q; ++q) {
      if (!enters(q)) continue;
      const R fq = fs[q];
      R val;
      if (mode == 0) {
        val = fq;
      } else if (mode == 1) {
        if (S == ILBM_STORAGE_F64)
          val = R(X::add(feq64_3<L>(q, rt64, ut64, vt64, wt64),
                         X::sub(double(fq), feq64_3<L>(q, r64, u64, v64, w64))));
        else
          val = R(feqs<L>(q, drt32, ut32, vt32, wt32) + (float(fq) - feqs<L>(q, dr32, u32, v32, w32)));
      } else {
        if (S == ILBM_STORAGE_F64)
          val = R(collide64_one<L>(q, double(fq), feq64<L>(q, r64, u64, v64, w64), a.tau, u64, v64,
                                   w64, double(gFx), double(gFy), double(gFz), ghf));
        else
          val = R(post32<L>(q, float(fq), col32_setup<L>(dr32, u32, v32, w32, a.om32, a.omh32,
                                                         float(gFx), float(gFy), float(gFz))));
      }
      Store<S>::store(fo + fidx(a, g[0] + L::cx(q), g[1] + L::cy(q), gk + L::cz(q)) + q * a.fs2, val,
                      sfac<L, S>(a, q));
    }
  }
}

// ---------------------------------------------------------------------------
// Main fused kernel
// ---------------------------------------------------------------------------
// Two forms.  The vector form (4- and 2-byte storage, rows that start on
// V-cell boundaries): a thread owns V consecutive columns of one row.  It
// loads its V cells of every population with one access, collides them two
// at a time in packed FP32 arithmetic, and stores one V-cell vector per
// population: the populations that land on its own columns, shifted along x
// by c_x with the missing cell taken from the neighbouring lane.  The first
// and last lane of a warp are halo lanes that collide their cells only for
// their neighbours (30 of 32 lanes own columns; the halo's loads hit L1 / L2),
// so no vector ever needs a cell of another warp.  The cell form (FP64, other
// layouts, and the rows on bounce-back walls): one cell per thread, one access
// per population.
//
// The bound is HBM; what keeps a form from it is the number of bytes in
// flight and the instructions per byte.  One cell per thread (64 registers, 32
// warps per SM) holds 78 KB of loads in flight per SM and issues 765 thread
// instructions per D3Q19 FP32 cell on rows whose x faces are periodic; four
// cells per thread (128 registers, 16 warps) hold 155 KB and issue 330, the
// arithmetic halved by the packed instructions and the address and index work
// shared by four cells.  Measured (B200): the 512 x 128 x 128 FP32 duct 313 ->
// 217 us per step (0.63 -> 0.92 of the copy bandwidth); the step alone, repeated, of
// the 256 x 128 x 128 level of the D3Q19 sphere 124 -> 104 us FP32 and 148 -> 94 us
// FP16, of the D3Q27 FP32 sphere 150 x 75 x 83 64 -> 48 us, of 2.1 M D3Q19 FP32
// cells 65 -> 57 us.
template <class L, int S>
struct StepVec {
  // 16 bytes per FP32 access; two cells for D3Q27, whose 27 populations of four
  // cells do not fit the registers; eight cells of FP16 spill (119 us against
  // 102 us for four in one build).  FP64 is bound by its arithmetic as well and stays with
  // one cell: two cells per thread spilled (437 against 389 us for two steps
  // of the 128 x 64 x 64 sphere).
  static constexpr int value = S == ILBM_STORAGE_F64 ? 1 : (L::Q <= 19 ? 4 : 2);
};

// blocks of kStepThreads resident per SM (the register target)
constexpr int kStepThreads = 128;
template <class L, int S, int V>
struct StepOcc {
  // (vector form: 128 registers for D3Q19, 80 for D2Q9, 96 for D3Q27; 160
  // registers and 12 warps measured 8% slower on the duct)
  static constexpr int value = S == ILBM_STORAGE_F64 ? (L::Q <= 9 ? 6 : 4)
                               : V == 4              ? (L::Q <= 9 ? 6 : 4)
                               : V == 2              ? 5
                                                     : (L::Q <= 9 ? 10 : L::Q <= 19 ? 8 : 5);
};

// a link that leaves through faces whose states are or-ed in m (AdvanceLBMAtLevel.cpp:272-373):
// reflected when every physical face it crosses is user_1 and no periodic one is crossed,
// delivered to its (wrapped) cell when nothing but wrapping faces are crossed, else dropped
constexpr int kFaceReturns = FACE_WRAP | FACE_REFLECT;
__device__ __forceinline__ bool link_reflects(int m) {
  return (m & FACE_REFLECT) && !(m & (FACE_WRAP | FACE_PHYS | FACE_PERIODIC));
}
__device__ __forceinline__ bool link_arrives(int m) { return !(m & ~FACE_WRAP); }

// ---- cell form ------------------------------------------------------------
// Cells whose row has a body force, stored macro fields or a face that
// returns populations take ANY; the others need none of its tests.  own /
// ownp / ownm: store the populations with c_x = 0 / +1 / -1 (a link returned
// by an x face counts as c_x = 0).
template <class L, int S, bool ANY>
__device__ __forceinline__ void step_cell(const StepArgs &a, int i, int j, int k, bool own, bool ownp,
                                          bool ownm) {
  using T = typename Store<S>::T;
  using R = typename Store<S>::R;
  const int64_t base = fidx(a, i, j, k);
  const T *fin = static_cast<const T *>(a.f_in) + base;
  R f[L::Q];
#pragma unroll
  for (int q = 0; q < L::Q; ++q) f[q] = Store<S>::load(fin + a.loff[q], a.sf[q]);
  R Fx = R(0), Fy = R(0), Fz = R(0), Px = R(0), Py = R(0), Pz = R(0);
  bool stored = false;
  if constexpr (ANY) {
    load_force<L, R>(a, a.force, i, j, k, Fx, Fy, Fz);
    load_force<L, R>(a, a.force_prev, i, j, k, Px, Py, Pz);
    stored = stored_macro_at(a, i, j, k);
  }
  // rho^n, u^n: stored, or recovered from f^n and F^{n-1}; then the collision in place
  if constexpr (S == ILBM_STORAGE_F64) {
    double rho, u, v, w;
    if (ANY && stored) {
      const int64_t m = midx(a, i, j, k);
      rho = ldm<double>(a.macro_in, m);
      u = ldm<double>(a.macro_in, m + a.ms2);
      v = ldm<double>(a.macro_in, m + 2 * a.ms2);
      w = (L::D == 3) ? ldm<double>(a.macro_in, m + 3 * a.ms2) : 0.0;
    } else {
      moments64_fast<L>(f, Px, Py, Pz, rho, u, v, w);
    }
    // the Guo increment is skipped where F == 0 (collide_forced.H:81-83)
    const bool hf = ANY && !(Fx == R(0) && Fy == R(0) && Fz == R(0));
    if (collide64_cell<L, ANY>(f, a.tau64, rho, u, v, w, Fx, Fy, Fz, hf)) {
      const double Pd[3] = {Px, Py, Pz}, Fd[3] = {Fx, Fy, Fz};
      double state[4] = {rho, u, v, w}, out[L::Q];
      collide64_redo<L>(fin, a.loff, a.tau, ANY && stored, Pd, Fd, state, out);
#pragma unroll
      for (int q = 0; q < L::Q; ++q) f[q] = out[q];
    }
  } else {
    float drho, u, v, w;
    if (ANY && stored) {
      const int64_t m = midx(a, i, j, k);
      drho = ldm<float>(a.macro_in, m) - 1.0f;
      u = ldm<float>(a.macro_in, m + a.ms2);
      v = ldm<float>(a.macro_in, m + 2 * a.ms2);
      w = (L::D == 3) ? ldm<float>(a.macro_in, m + 3 * a.ms2) : 0.0f;
    } else {
      moments32<L>(f, Px, Py, Pz, drho, u, v, w);
    }
    const Col32 c = col32_setup<L>(drho, u, v, w, a.om32, a.omh32, Fx, Fy, Fz);
#pragma unroll
    for (int q = 0; q < L::Q; ++q) f[q] = post32<L>(q, f[q], c);
  }
  // Push f*(y,q) to y + c_q.  Populations that leave the box through a face
  // that does not return them land in the ghost layer of f_out (scratch,
  // never read), or are not stored.
  T *fob = static_cast<T *>(a.f_out) + base;
  bool edge = false;
  if constexpr (ANY)
    edge = i == a.lo[0] || i == a.hi[0] || j == a.lo[1] || j == a.hi[1] ||
           (L::D == 3 && (k == a.lo[2] || k == a.hi[2]));
  if (!edge) {
#pragma unroll
    for (int q = 0; q < L::Q; ++q)
      if (L::cx(q) == 0 ? own : (L::cx(q) > 0 ? ownp : ownm)) fob[a.doff[q]] = Store<S>::pack(f[q], a.sf[q]);
    return;
  }
  const int st[3][2] = {{i == a.lo[0] ? a.face_lo[0] : 0, i == a.hi[0] ? a.face_hi[0] : 0},
                        {j == a.lo[1] ? a.face_lo[1] : 0, j == a.hi[1] ? a.face_hi[1] : 0},
                        {L::D == 3 && k == a.lo[2] ? a.face_lo[2] : 0, L::D == 3 && k == a.hi[2] ? a.face_hi[2] : 0}};
  const int64_t span[3] = {(int64_t)(a.hi[0] - a.lo[0] + 1), (int64_t)(a.hi[1] - a.lo[1] + 1) * a.fs0,
                           (int64_t)(a.hi[2] - a.lo[2] + 1) * a.fs1};
#pragma unroll
  for (int q = 0; q < L::Q; ++q) {
    const int c[3] = {L::cx(q), L::cy(q), L::cz(q)};
    int m = 0;
    int64_t wrap = 0;
#pragma unroll
    for (int d = 0; d < L::D; ++d) {
      if (c[d] == 0) continue;
      const int s = st[d][c[d] > 0];
      m |= s;
      if (s == FACE_WRAP) wrap += c[d] > 0 ? -span[d] : span[d];
    }
    const bool returned = c[0] != 0 && st[0][c[0] > 0] != 0;
    if (!((c[0] == 0 || returned) ? own : (c[0] > 0 ? ownp : ownm))) continue;
    if (link_reflects(m))
      fob[a.loff[opposite<L>(q)]] = Store<S>::pack(f[q], a.sf[opposite<L>(q)]);
    else if (link_arrives(m))
      fob[a.doff[q] + wrap] = Store<S>::pack(f[q], a.sf[q]);
  }
}

// a row piece [x0, x1] of (j, k) that needs ANY: rows on a face that returns
// populations, and rows on any face when an x face does (x_too: the piece's
// own x faces as well); stored macro fields; force arrays or a uniform force
template <class L>
__device__ __forceinline__ bool needs_any(const StepArgs &a, int x0, int x1, int j, int k, bool x_too) {
  const int fs = (j == a.lo[1] ? a.face_lo[1] : 0) | (j == a.hi[1] ? a.face_hi[1] : 0) |
                 (L::D == 3 && k == a.lo[2] ? a.face_lo[2] : 0) | (L::D == 3 && k == a.hi[2] ? a.face_hi[2] : 0);
  if (fs && ((fs | a.face_lo[0] | a.face_hi[0]) & kFaceReturns)) return true;
  if (x_too && ((x0 == a.lo[0] && (a.face_lo[0] & kFaceReturns)) ||
                (x1 >= a.hi[0] && (a.face_hi[0] & kFaceReturns))))
    return true;
  if (a.macro_in &&
      (!a.use_mbox || (j >= a.mblo[1] && j <= a.mbhi[1] && (L::D == 2 || (k >= a.mblo[2] && k <= a.mbhi[2])) &&
                       x1 >= a.mblo[0] && x0 <= a.mbhi[0])))
    return true;
  if (a.force == nullptr || a.force_prev == nullptr) return a.force != a.force_prev;
  return j >= a.flo[1] && j <= a.fhi[1] && (L::D == 2 || (k >= a.flo[2] && k <= a.fhi[2])) && x1 >= a.flo[0] &&
         x0 <= a.fhi[0];
}

__device__ __forceinline__ bool in_skip(const StepArgs &a, int D, int j, int k) {
  return a.use_skip && j >= a.slo[1] && j <= a.shi[1] && (D == 2 || (k >= a.slo[2] && k <= a.shi[2]));
}

// ---- vector form ------------------------------------------------------------
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

// V consecutive populations, loaded and stored in one access and held in
// registers as pairs in their storage form (4-byte: two floats, 2-byte: one
// half2, converted when the pair is collided).  s / si: the direction's
// storage factor and its inverse, rounded to nearest.
template <int B>
struct Bytes;
template <>
struct Bytes<4> { using type = unsigned; };
template <>
struct Bytes<8> { using type = uint2; };
template <>
struct Bytes<16> { using type = uint4; };

template <int S>
struct VecPair;
template <>
struct VecPair<ILBM_STORAGE_F32_SHIFT> {
  using Raw = float2;
  __device__ static __forceinline__ Raw zero() { return f2(0.0f); }
  __device__ static __forceinline__ float2 get(Raw r, float) { return r; }
  __device__ static __forceinline__ Raw put(float2 v, float, float) { return v; }
  // the pair (b's second, c's first)
  __device__ static __forceinline__ Raw join(Raw b, Raw c) { return make_float2(b.y, c.x); }
  __device__ static __forceinline__ Raw from_up(Raw last) {  // the lane below's last cell, in second place
    return make_float2(0.0f, __shfl_up_sync(0xffffffffu, last.y, 1));
  }
  __device__ static __forceinline__ Raw from_down(Raw first) {  // the lane above's first cell, in first place
    return make_float2(__shfl_down_sync(0xffffffffu, first.x, 1), 0.0f);
  }
  __device__ static __forceinline__ float cell(Raw r, int e) { return e ? r.y : r.x; }
};
template <>
struct VecPair<ILBM_STORAGE_F16_SCALED> {
  using Raw = unsigned;
  __device__ static __forceinline__ Raw zero() { return 0u; }
  __device__ static __forceinline__ float2 get(Raw r, float s) {
    return __fmul2_rn(__half22float2(*reinterpret_cast<const __half2 *>(&r)), f2(s));
  }
  // v / s rounded as the division rounds it: q = v * si, then one Markstein
  // correction (exact for every 24-bit v with si the nearest 1 / s).  Both
  // signs of zero come out as the division's; v is held to 1e20, which any
  // scale that vec_width() lets through still takes to infinity, so that an infinite v
  // does not meet itself in the remainder; NaN stays.
  __device__ static __forceinline__ Raw put(float2 v, float s, float si) {
    v = make_float2(held(v.x), held(v.y));
    const float2 q = __fmul2_rn(v, f2(si));
    const float2 r = __ffma2_rn(q, f2(s), make_float2(-v.x, -v.y));
    const __half2 h = __float22half2_rn(__ffma2_rn(r, f2(-si), q));
    return *reinterpret_cast<const unsigned *>(&h);
  }
  __device__ static __forceinline__ float held(float v) {
    float m;
    asm("min.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(m) : "f"(v), "f"(1e20f));
    return m;
  }
  __device__ static __forceinline__ Raw join(Raw b, Raw c) { return __byte_perm(b, c, 0x5432); }
  __device__ static __forceinline__ Raw from_up(Raw last) { return __shfl_up_sync(0xffffffffu, last, 1); }
  __device__ static __forceinline__ Raw from_down(Raw first) { return __shfl_down_sync(0xffffffffu, first, 1); }
  __device__ static __forceinline__ __half cell(Raw r, int e) {
    return __ushort_as_half((unsigned short)(e ? r >> 16 : r & 0xffffu));
  }
};

template <int S, int V>
struct Vec {
  using T = typename Store<S>::T;
  using P = VecPair<S>;
  using Raw = typename P::Raw;
  static constexpr int N = V / 2;
  // the first n elements' access, n a power of two up to V
  template <int n>
  __device__ static __forceinline__ void store_some(T *p, const Raw *v) {
    using W = typename Bytes<n * (int)sizeof(T)>::type;
    union {
      W w;
      Raw r[n / 2];
    } u;
#pragma unroll
    for (int h = 0; h < n / 2; ++h) u.r[h] = v[h];
    *reinterpret_cast<W *>(p) = u.w;
  }
  __device__ static __forceinline__ void load(const T *p, Raw (&v)[N]) {
    using W = typename Bytes<V * (int)sizeof(T)>::type;
    union {
      W w;
      Raw r[N];
    } u;
    u.w = __ldg(reinterpret_cast<const W *>(p));
#pragma unroll
    for (int h = 0; h < N; ++h) v[h] = u.r[h];
  }
  __device__ static __forceinline__ void store(T *p, const Raw (&v)[N]) { store_some<V>(p, v); }
  // all but the first / the last element
  __device__ static __forceinline__ void store_nofirst(T *p, const Raw (&v)[N]) {
    p[1] = P::cell(v[0], 1);
    if constexpr (V >= 4) store_some<2>(p + 2, v + 1);
    if constexpr (V >= 8) store_some<4>(p + 4, v + 2);
  }
  __device__ static __forceinline__ void store_nolast(T *p, const Raw (&v)[N]) {
    if constexpr (V >= 8) store_some<4>(p, v);
    if constexpr (V >= 4) store_some<2>(p + V - 4, v + N - 2);
    p[V - 2] = P::cell(v[N - 1], 0);
  }
};

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.0f), a); }  // exact product
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// c'.x of the canonical member of q's pair (canon_dot) for two cells
template <class L>
__device__ __forceinline__ float2 canon_dot2(int q, float2 x, float2 y, float2 z) {
  const int s = pair_sign<L>(q);
  const int c[3] = {s * L::cx(q), s * L::cy(q), s * L::cz(q)};
  const float2 v[3] = {x, y, z};
  float2 r = f2(0.0f);
  bool first = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (c[d] == 0) continue;
    r = first ? v[d] : (c[d] > 0 ? add2(r, v[d]) : sub2(r, v[d]));  // the first one is +1
    first = false;
  }
  return r;
}

// what a warp's vectors carry beyond their populations
enum VecMode {
  VEC_PLAIN = 0,   // nothing
  VEC_FORCED = 1,  // a uniform force on the level
  VEC_DATA = 2     // anything: force arrays, stored macro fields, wrapped rows
};

// F^n, F^{n-1} and the stored rho, u of two cells (where st is set)
struct PairData {
  float2 F[3], P[3], mac[4];
  bool st[2];
};

// moments32, col32_setup and post32 for two cells at once: the same roundings
// in the same order, so the results are those of the cell form (which skips
// the Guo increment where F = 0; here it then adds a zero).
template <class L, int MODE>
__device__ __forceinline__ void collide_pair(const StepArgs &a, const PairData &d, float2 (&g)[L::Q]) {
  constexpr bool F_ON = MODE != VEC_PLAIN;
  float2 r = f2(0.0f), m[3] = {f2(0.0f), f2(0.0f), f2(0.0f)};
#pragma unroll
  for (int q = 0; q < L::Q; ++q) {
    const int c[3] = {L::cx(q), L::cy(q), L::cz(q)};
    r = add2(r, g[q]);
#pragma unroll
    for (int e = 0; e < 3; ++e)
      if (c[e]) m[e] = c[e] > 0 ? add2(m[e], g[q]) : sub2(m[e], g[q]);
  }
  const float2 sum = add2(f2(1.0f), r);
  const float2 inv = make_float2(__fdiv_rn(1.0f, sum.x), __fdiv_rn(1.0f, sum.y));
  float2 u[3];
#pragma unroll
  for (int e = 0; e < 3; ++e)
    u[e] = (e < L::D) ? mul2(F_ON ? fma2(f2(0.5f), d.P[e], m[e]) : m[e], inv) : f2(0.0f);
  if (MODE == VEC_DATA) {
    if (d.st[0]) {
      r.x = __fsub_rn(d.mac[0].x, 1.0f);
#pragma unroll
      for (int e = 0; e < L::D; ++e) u[e].x = d.mac[1 + e].x;
    }
    if (d.st[1]) {
      r.y = __fsub_rn(d.mac[0].y, 1.0f);
#pragma unroll
      for (int e = 0; e < L::D; ++e) u[e].y = d.mac[1 + e].y;
    }
  }
  const float om = a.om32, omh = a.omh32;
  const float2 m15uu = mul2(f2(-1.5f), fma2(u[2], u[2], fma2(u[1], u[1], mul2(u[0], u[0]))));
  const float2 omd = mul2(f2(om), r), omr = mul2(f2(om), add2(f2(1.0f), r));
  const float2 omm = f2(__fsub_rn(1.0f, om));
  const float2 m3uF =
      F_ON ? mul2(f2(-3.0f), fma2(u[2], d.F[2], fma2(u[1], d.F[1], mul2(u[0], d.F[0])))) : f2(0.0f);
#pragma unroll
  for (int q = 0; q < L::Q; ++q) {
    const int o = opposite<L>(q);
    if (o < q) continue;  // done with its pair
    const float wq = float(L::w(q));
    const float2 omrw = mul2(omr, f2(wq)), omdw = mul2(omd, f2(wq));
    const float woh = __fmul_rn(wq, omh);
    if (o == q) {  // the rest direction
      float2 b = fma2(omrw, m15uu, omdw);
      if (F_ON) b = fma2(f2(woh), m3uF, b);
      g[q] = fma2(omm, g[q], b);
      continue;
    }
    const float2 cu = canon_dot2<L>(q, u[0], u[1], u[2]);
    const float2 t = fma2(mul2(f2(4.5f), cu), cu, m15uu);
    float2 b = fma2(omrw, t, omdw);
    float2 p = mul2(mul2(f2(3.0f), omrw), cu);
    if (F_ON) {
      const float2 cF = canon_dot2<L>(q, d.F[0], d.F[1], d.F[2]);
      b = fma2(f2(woh), fma2(mul2(f2(9.0f), cu), cF, m3uF), b);
      p = fma2(f2(__fmul_rn(3.0f, woh)), cF, p);
    }
    const int up = pair_sign<L>(q) > 0 ? q : o, dn = pair_sign<L>(q) > 0 ? o : q;
    g[up] = fma2(omm, g[up], add2(b, p));
    g[dn] = fma2(omm, g[dn], sub2(b, p));
  }
}

// the data of cells i, i + 1 of (j, k); act: which of them exist
template <class L>
__device__ __forceinline__ PairData pair_data(const StepArgs &a, int i, int j, int k, uint32_t act) {
  PairData d;
  float F[2][3], P[2][3], M[2][4];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    F[e][0] = F[e][1] = F[e][2] = P[e][0] = P[e][1] = P[e][2] = 0.0f;
    M[e][0] = M[e][1] = M[e][2] = M[e][3] = 0.0f;
    d.st[e] = false;
    if (!((act >> e) & 1u)) continue;
    load_force<L, float>(a, a.force, i + e, j, k, F[e][0], F[e][1], F[e][2]);
    load_force<L, float>(a, a.force_prev, i + e, j, k, P[e][0], P[e][1], P[e][2]);
    d.st[e] = stored_macro_at(a, i + e, j, k);
    if (d.st[e]) {
      const int64_t m = midx(a, i + e, j, k);
#pragma unroll
      for (int c = 0; c <= L::D; ++c) M[e][c] = ldm<float>(a.macro_in, m + c * a.ms2);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const bool z = c == 2 && L::D != 3;  // (a 2D lattice has no third force component)
    d.F[c] = z ? f2(0.0f) : make_float2(F[0][c], F[1][c]);
    d.P[c] = z ? f2(0.0f) : make_float2(P[0][c], P[1][c]);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) d.mac[c] = make_float2(M[0][c], M[1][c]);
  return d;
}

// the destination vector at the thread's columns of a population that moves
// by c along x: the missing cell comes from the neighbouring lane
template <int S, int V>
__device__ __forceinline__ void shifted(const typename Vec<S, V>::Raw (&g)[V / 2], int c,
                                        typename Vec<S, V>::Raw (&s)[V / 2]) {
  using P = VecPair<S>;
  constexpr int N = V / 2;
  if (c > 0) {
    const auto e = P::from_up(g[N - 1]);
#pragma unroll
    for (int h = 0; h < N; ++h) s[h] = P::join(h ? g[h - 1] : e, g[h]);
  } else if (c < 0) {
    const auto e = P::from_down(g[0]);
#pragma unroll
    for (int h = 0; h < N; ++h) s[h] = P::join(g[h], h + 1 < N ? g[h + 1] : e);
  } else {
#pragma unroll
    for (int h = 0; h < N; ++h) s[h] = g[h];
  }
}

// The vector form.  act: the lane's cells that this launch owns; mz / mp / mm:
// the elements of the thread's columns that populations with c_x = 0 / +1 / -1
// arrive at (0 for halo lanes); xlo / xhi: element of the box's first / last
// column whose links an x face returns (-1: none).  Every lane of the warp
// calls it.
template <class L, int S, int V, int MODE>
__device__ __forceinline__ void step_vector(const StepArgs &a, int x0, int j, int k, uint32_t act, uint32_t mz,
                                            uint32_t mp, uint32_t mm, int xlo, int xhi) {
  using T = typename Store<S>::T;
  constexpr uint32_t ALL = (1u << V) - 1u, NOFIRST = ALL & ~1u, NOLAST = ALL >> 1;
  const int64_t base = fidx(a, x0, j, k);
  using P = VecPair<S>;
  typename P::Raw f[L::Q][V / 2];
  {
    // (a vector may reach V - 1 cells past its row: the next row's memory)
    const T *fin = static_cast<const T *>(a.f_in) + base;
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      if (act) {
        Vec<S, V>::load(fin + a.loff[q], f[q]);
      } else {
#pragma unroll
        for (int h = 0; h < V / 2; ++h) f[q][h] = P::zero();
      }
    }
  }
#pragma unroll
  for (int h = 0; h < V / 2; ++h) {
    float2 g[L::Q];
#pragma unroll
    for (int q = 0; q < L::Q; ++q) g[q] = P::get(f[q][h], a.sf[q]);
    PairData d;
    if (MODE == VEC_DATA) {
      d = pair_data<L>(a, x0 + 2 * h, j, k, act >> (2 * h));
    } else if (MODE == VEC_FORCED) {
#pragma unroll
      for (int c = 0; c < 3; ++c) d.F[c] = d.P[c] = f2(c < L::D ? float(a.uf[c]) : 0.0f);
    }
    collide_pair<L, MODE>(a, d, g);
#pragma unroll
    for (int q = 0; q < L::Q; ++q) f[q][h] = P::put(g[q], a.sf[q], a.si[q]);
  }
  // rows on a wrapping face deliver to the opposite row
  int64_t yw[2] = {0, 0}, zw[2] = {0, 0};
  int ys[2] = {0, 0}, zs[2] = {0, 0};
  if (MODE == VEC_DATA) {
    if (j == a.lo[1]) ys[0] = a.face_lo[1];
    if (j == a.hi[1]) ys[1] = a.face_hi[1];
    if (ys[0] == FACE_WRAP) yw[0] = (int64_t)(a.hi[1] - a.lo[1] + 1) * a.fs0;
    if (ys[1] == FACE_WRAP) yw[1] = -(int64_t)(a.hi[1] - a.lo[1] + 1) * a.fs0;
    if (L::D == 3) {
      if (k == a.lo[2]) zs[0] = a.face_lo[2];
      if (k == a.hi[2]) zs[1] = a.face_hi[2];
      if (zs[0] == FACE_WRAP) zw[0] = (int64_t)(a.hi[2] - a.lo[2] + 1) * a.fs1;
      if (zs[1] == FACE_WRAP) zw[1] = -(int64_t)(a.hi[2] - a.lo[2] + 1) * a.fs1;
    }
  }
  auto row_wrap = [&](int q) -> int64_t {
    int64_t o = 0;
    if (MODE == VEC_DATA) {
      if (L::cy(q)) o += yw[L::cy(q) > 0];
      if (L::cz(q)) o += zw[L::cz(q) > 0];
    }
    return o;
  };
  auto row_state = [&](int q) -> int {
    int s = 0;
    if (MODE == VEC_DATA) {
      if (L::cy(q)) s |= ys[L::cy(q) > 0];
      if (L::cz(q)) s |= zs[L::cz(q) > 0];
    }
    return s;
  };
  T *fob = static_cast<T *>(a.f_out) + base;
  const bool regular = (mz == ALL || mz == 0) && (mp == ALL || mp == 0 || mp == NOFIRST) &&
                       (mm == ALL || mm == 0 || mm == NOLAST);
  if (MODE != VEC_DATA && __all_sync(0xffffffffu, regular)) {
    // whole vectors, or all but the cell that comes from outside the box
    const bool wz = mz == ALL, wp = mp == ALL, wm = mm == ALL, ep = mp == NOFIRST, em = mm == NOLAST;
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      const int cx = L::cx(q);
      T *dst = fob + (a.doff[q] - cx);
      typename P::Raw s[V / 2];
      shifted<S, V>(f[q], cx, s);
      if (cx == 0 ? wz : (cx > 0 ? wp : wm)) Vec<S, V>::store(dst, s);
      if (cx > 0 && ep) Vec<S, V>::store_nofirst(dst, s);
      if (cx < 0 && em) Vec<S, V>::store_nolast(dst, s);
    }
  } else {
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      const int cx = L::cx(q);
      T *dst = fob + (a.doff[q] - cx + row_wrap(q));
      const uint32_t m = cx == 0 ? mz : (cx > 0 ? mp : mm);
      typename P::Raw s[V / 2];
      shifted<S, V>(f[q], cx, s);
      if (m == ALL) {
        Vec<S, V>::store(dst, s);
      } else {
#pragma unroll
        for (int e = 0; e < V; ++e)
          if ((m >> e) & 1u) dst[e] = P::cell(s[e / 2], e & 1);
      }
    }
  }
  if (__any_sync(0xffffffffu, xlo >= 0 || xhi >= 0)) {
    const int nx = a.hi[0] - a.lo[0] + 1;
#pragma unroll
    for (int q = 0; q < L::Q; ++q) {
      const int cx = L::cx(q);
      if (cx == 0) continue;
      const int e = cx > 0 ? xhi : xlo;
      if (e < 0) continue;
      const int face = cx > 0 ? a.face_hi[0] : a.face_lo[0], s = face | row_state(q);
      T v = P::cell(f[q][0], 0);
#pragma unroll
      for (int h = 1; h < V; ++h)
        if (e == h) v = P::cell(f[q][h / 2], h & 1);
      if (link_arrives(s))
        fob[a.doff[q] + row_wrap(q) + e + (cx > 0 ? -nx : nx)] = v;
      else if (link_reflects(s))  // (w_q = w_{q_bar}: the same storage factor)
        fob[a.loff[opposite<L>(q)] + e] = v;
    }
  }
}

// warp w of a launch: vectors kOwned w - 1 .. kOwned w + 30 of the sequence (row
// v / vpr of the region, j fastest; the vectors of a row in order)
template <class L, int S, int V>
__device__ __forceinline__ void step_warp(const StepArgs &a, uint32_t w) {
  constexpr uint32_t ALL = (1u << V) - 1u;
  const int lane = threadIdx.x & 31;
  const uint32_t v = w * kOwned + (uint32_t)lane - 1u;  // (-1 wraps: past the end)
  const bool valid = v < a.nvec;
  const uint32_t row = fast_div(valid ? v : 0u, a.dvpr);
  const uint32_t p = valid ? v - row * a.vpr : 0u;
  const uint32_t kk = (L::D == 3) ? fast_div(row, a.dvny) : 0u;
  const int j = a.rlo[1] + (int)(row - kk * a.vny), k = a.rlo[2] + (int)kk;
  const int x0 = a.vx0 + (int)p * V;
  uint32_t act = 0;  // the cells this launch owns
  if (valid) {
    const int e0 = max(a.rlo[0] - x0, 0), e1 = min(a.rhi[0] - x0, V - 1);
    if (e0 <= e1) act = ((2u << e1) - 1u) & ~((1u << e0) - 1u);
    if (in_skip(a, L::D, j, k)) {
      const int s0 = max(a.slo[0] - x0, 0), s1 = min(a.shi[0] - x0, V - 1);
      if (s0 <= s1) act &= ~(((2u << s1) - 1u) & ~((1u << s0) - 1u));
    }
  }
  if (!__any_sync(0xffffffffu, act != 0)) return;
  uint32_t prev = __shfl_up_sync(0xffffffffu, act, 1), next = __shfl_down_sync(0xffffffffu, act, 1);
  if (lane == 0 || p == 0) prev = 0;
  if (lane == 31 || p + 1 == a.vpr) next = 0;
  const bool owner = valid && lane >= 1 && lane <= kOwned;
  const bool wall = act && ((j == a.lo[1] && a.face_lo[1] == FACE_REFLECT) ||
                            (j == a.hi[1] && a.face_hi[1] == FACE_REFLECT) ||
                            (L::D == 3 && ((k == a.lo[2] && a.face_lo[2] == FACE_REFLECT) ||
                                           (k == a.hi[2] && a.face_hi[2] == FACE_REFLECT))));
  if (__any_sync(0xffffffffu, wall)) {
    // rows that reflect: the window's cells one by one, consecutive lanes on consecutive cells;
    // each stores what lands on the warp's own columns
#pragma unroll 1
    for (int it = 0; it < V; ++it) {
      const int c = it * 32 + lane, from = c / V, e = c % V;
      const int cx0 = __shfl_sync(0xffffffffu, x0, from), cj = __shfl_sync(0xffffffffu, j, from);
      const int ck = __shfl_sync(0xffffffffu, k, from);
      const uint32_t cact = __shfl_sync(0xffffffffu, act, from);
      if (!((cact >> e) & 1u)) continue;
      const int up = e == V - 1 ? from + 1 : from, dn = e == 0 ? from - 1 : from;
      step_cell<L, S, true>(a, cx0 + e, cj, ck, from >= 1 && from <= kOwned, up >= 1 && up <= kOwned,
                            dn >= 1 && dn <= kOwned);
    }
    return;
  }
  uint32_t mz = 0, mp = 0, mm = 0;
  int xlo = -1, xhi = -1;
  if (owner) {
    const int ehi = a.hi[0] - x0;  // element of the box's last column
    const uint32_t in = ehi >= V - 1 ? ALL : ((2u << ehi) - 1u);
    mz = act;
    mp = ((act << 1) | (prev >> (V - 1))) & in;
    mm = ((act >> 1) | ((next & 1u) << (V - 1))) & in;
    if (x0 == a.lo[0] && (act & 1u) && (a.face_lo[0] & kFaceReturns)) xlo = 0;
    if (ehi >= 0 && ehi < V && ((act >> ehi) & 1u) && (a.face_hi[0] & kFaceReturns)) xhi = ehi;
  }
  // (of a vector cut by the skip box only the cells outside it count)
  const int xa = x0 + __ffs(act) - 1, xb = x0 + 31 - __clz(act);
  if (__any_sync(0xffffffffu, act && needs_any<L>(a, xa, xb, j, k, false)))
    step_vector<L, S, V, VEC_DATA>(a, x0, j, k, act, mz, mp, mm, xlo, xhi);
  else if (a.forced)
    step_vector<L, S, V, VEC_FORCED>(a, x0, j, k, act, mz, mp, mm, xlo, xhi);
  else
    step_vector<L, S, V, VEC_PLAIN>(a, x0, j, k, act, mz, mp, mm, xlo, xhi);
}

// cell c of a launch in the cell form
template <class L, int S>
__device__ __forceinline__ void step_single(const StepArgs &a, uint32_t c) {
  if (c >= a.nvec) return;
  const uint32_t row = fast_div(c, a.dvpr);
  const uint32_t kk = (L::D == 3) ? fast_div(row, a.dvny) : 0u;
  const int i = a.vx0 + (int)(c - row * a.vpr);
  const int j = a.rlo[1] + (int)(row - kk * a.vny), k = a.rlo[2] + (int)kk;
  if (in_skip(a, L::D, j, k) && i >= a.slo[0] && i <= a.shi[0]) return;
  if (a.forced || needs_any<L>(a, i, i, j, k, true))
    step_cell<L, S, true>(a, i, j, k, true, true, true);
  else
    step_cell<L, S, false>(a, i, j, k, true, true, true);
}

template <class L, int S, int V>
__device__ __forceinline__ void step_block(const StepArgs &a, uint32_t first) {
  if constexpr (V > 1)
    step_warp<L, S, V>(a, first / kOwned + (threadIdx.x >> 5));
  else
    step_single<L, S>(a, first + threadIdx.x);
}

// Block b of a box: every ghost_every-th of the leading blocks pushes the ghost
// shell's populations (ghost_push, one ghost cell per thread); the rest take the
// cells.  (All ghost blocks first filled the SMs with scattered accesses before
// the streaming started.)
template <class L, int S, int V>
__device__ __forceinline__ void step_or_ghosts(const StepArgs &a, const int (*lb)[6], uint32_t b) {
  if (a.ghost_blocks) {
    const uint32_t g = fast_div(b, a.dghost);
    if (g < a.ghost_blocks && g * a.ghost_every == b) {
      ghost_push<L, S>(a, lb, g * kStepThreads + threadIdx.x, a.ghost_blocks * kStepThreads);
      return;
    }
    b -= min(g + 1u, a.ghost_blocks);
  }
  step_block<L, S, V>(a, b * step_vectors_per_block(V, kStepThreads));
}

template <class L, int S, int V>
__global__ void __launch_bounds__(kStepThreads, StepOcc<L, S, V>::value)
    k_step(const __grid_constant__ StepArgs a) {
  step_or_ghosts<L, S, V>(a, &a.lb0, blockIdx.x);
}

// The boxes of a level in one launch: a box's last blocks run beside the next
// box's, where a launch per box left the device idle at each end (twelve
// 50 x 50 x 45 FP64 boxes with their macro fields: 297 -> 191 us).
template <class L, int S, int V>
__global__ void __launch_bounds__(kStepThreads, StepOcc<L, S, V>::value)
    k_step_boxes(const __grid_constant__ StepBoxes p) {
  int n = 0;
  while (n + 1 < p.nbox && blockIdx.x >= p.first[n + 1]) ++n;
  step_or_ghosts<L, S, V>(p.a[n], p.lb.lb, blockIdx.x - p.first[n]);
}

// ---------------------------------------------------------------------------
// Batched level step: many independent cases (each one box = its level
// domain, self-filled ghosts) in one persistent launch.  Blocks walk a tile
// table of vector runs and ghost-push chunks over all cases; the arguments
// of a tile's case are copied to shared memory, so the per-direction offsets
// stay on chip and cannot alias the population stores.
// ---------------------------------------------------------------------------
template <class L, int S, int V>
struct BatchOcc {
  static constexpr int value = (StepOcc<L, S, V>::value * kStepThreads) / 256;
};

template <class L, int S, int V>
__global__ void __launch_bounds__(256, BatchOcc<L, S, V>::value)
    k_step_batch(const StepArgs *__restrict__ args, const StepTile *__restrict__ tiles, int ntiles,
                 const int *steps, const int *limit) {
  __shared__ StepArgs sa;
  int cur = -1;  // every thread walks the same tiles, so this stays block-uniform
  // strided over the table (block b takes entries b, b + gridDim.x, ...),
  // which the batch lays out so that the blocks in flight stream through
  // neighbouring rows together (a contiguous run of rows per block measured
  // 2.2x slower: the push stores' split lines no longer meet in L2) while a
  // block keeps to one case; c = -1 marks a filler entry
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const StepTile tl = tiles[t];
    if (tl.c < 0 || steps[tl.c] >= limit[tl.c]) continue;  // filler, or a case that has taken all its steps
    if (tl.c != cur) {
      __syncthreads();  // every thread is done with the previous case's arguments
      const int *src = reinterpret_cast<const int *>(args + tl.c);
      int *dst = reinterpret_cast<int *>(&sa);
      for (int w = threadIdx.x; w < (int)(sizeof(StepArgs) / sizeof(int)); w += blockDim.x)
        dst[w] = src[w];
      __syncthreads();
      cur = tl.c;
    }
    if (tl.ghosts)
      ghost_push<L, S>(sa, &sa.lb0, tl.first + threadIdx.x, tl.ghosts);
    else
      step_block<L, S, V>(sa, tl.first);
  }
}

// the cells a thread of the level step takes at once: StepVec where every
// row of both population arrays starts on that many cells, else 1
template <class L, int S>
int vec_width(const StepArgs &a) {
  using T = typename Store<S>::T;
  constexpr int V = StepVec<L, S>::value;
  const int64_t off = (int64_t)(a.lo[0] - a.fgl[0]) + (int64_t)(a.lo[1] - a.fgl[1]) * a.fs0 +
                      (int64_t)(a.lo[2] - a.fgl[2]) * a.fs1;
  const uintptr_t in = (uintptr_t)(static_cast<const T *>(a.f_in) + off);
  const uintptr_t out = (uintptr_t)(static_cast<const T *>(a.f_out) + off);
  const bool ok = in % (V * sizeof(T)) == 0 && out % (V * sizeof(T)) == 0 && a.fs0 % V == 0 &&
                  a.fs2 % V == 0 && (L::D == 2 || a.fs1 % V == 0);
  // F16: VecPair's division wants a scale within 2^-40 .. 2^40 (si is about
  // two to three times it); any other takes the cell form, which divides
  const bool scale_ok = S != ILBM_STORAGE_F16_SCALED || (a.si[0] > 0x1p-38f && a.si[0] < 0x1p40f);
  return ok && scale_ok ? V : 1;
}

// the blocks of a planned launch; with ghost_blocks set, those of the ghost
// shell's push among them
static uint32_t plan_blocks(StepArgs &a, int V) {
  const uint32_t per = step_vectors_per_block(V, kStepThreads), cells = (a.nvec + per - 1) / per;
  if (a.ghost_blocks) {
    a.ghost_blocks = std::min(1u << 20, (a.goff[3] + kStepThreads - 1) / kStepThreads);
    if (a.ghost_blocks) {
      a.ghost_every = 1 + cells / a.ghost_blocks;
      a.dghost = div_magic(a.ghost_every);
    }
  }
  return a.ghost_blocks + cells;
}

// k_step over [rlo, rhi] (minus the skip box), with the ghost shell push in
// leading blocks when with_ghosts is set
template <class L, int S, int V>
static void launch_vectors(ilbm_ctx *ctx, const StepArgs &a_in, cudaStream_t st, bool with_ghosts) {
  StepArgs a = a_in;
  const int e = L::D - 1;  // a region of 2^30 vectors or more goes in slices along the last dimension
  const int64_t slice = (int64_t)((a.rhi[0] - a.rlo[0]) / V + 2) * (L::D == 3 ? a.rhi[1] - a.rlo[1] + 1 : 1);
  const int64_t most = std::max<int64_t>(1, (int64_t)(1 << 30) / std::max<int64_t>(1, slice));
  const int last = a.rhi[e];
  for (int64_t s = a.rlo[e]; s <= last; s += most) {
    a.rlo[e] = (int)s;
    a.rhi[e] = (int)std::min<int64_t>(last, s + most - 1);
    if (!plan_vectors(a, L::D, V)) return;
    a.ghost_blocks = with_ghosts ? 1u : 0u;
    with_ghosts = false;
    const uint32_t blocks = plan_blocks(a, V);
    k_step<L, S, V><<<blocks, kStepThreads, 0, st>>>(a);
    ctx->launches++;
  }
}

// Launches that the cell form takes in rows that start on vectors too (B200, us
// per level step, vector / cell form):
//   - few cells, whose time is one thread's chain and not the traffic.  With a
//     reflecting y or z face a warp of the vector form walks its cells one after
//     another: up to 2^17 cells (D2Q9 98k 8.2 / 6.2 FP32, 9.1 / 6.2 FP16; D3Q19
//     131k 12.4 / 9.3 and 18.5 / 12.4; D3Q27 131k 12.4 / 12.4 and 18.4 / 18.2, and at
//     393k 24.1 / 24.3 and 32.2 / 39.1).  Without one, FP32 up to 2^15 cells (D2Q9 25k
//     6.2 / 4.3, D3Q19 33k 8.3 / 6.2, D3Q27 9.3 / 6.2; with a flow's ghost shell D3Q19
//     33k 10.3 / 10.1, 61k 9.3 / 10.3); the FP16 vectors' fewer accesses win from
//     the start (D3Q27 15k 8.3 / 10.0)
//   - D3Q19 FP32 with stored macro fields and force arrays on every cell, eleven
//     scattered loads per cell (2.4 M cells 100 / 91)
//   - a body's band (singly), where every cell reads force arrays: 23 against 28
//     us for the 358k cells of the two-level sphere's band
template <class L, int S>
static bool prefers_cells(const StepArgs &a) {
  int64_t cells = 1;
  bool wall = false, all_forced = a.macro_in && !a.use_mbox && a.force;
  for (int d = 0; d < L::D; ++d) {
    cells *= a.rhi[d] - a.rlo[d] + 1;
    if (d > 0) wall = wall || a.face_lo[d] == FACE_REFLECT || a.face_hi[d] == FACE_REFLECT;
    all_forced = all_forced && a.flo[d] <= a.rlo[d] && a.fhi[d] >= a.rhi[d];
  }
  if (cells <= (wall ? 1 << 17 : (S == ILBM_STORAGE_F32_SHIFT ? 1 << 15 : 0))) return true;
  return L::Q == 19 && S == ILBM_STORAGE_F32_SHIFT && all_forced;
}

template <class L, int S>
void launch_cells(ilbm_ctx *ctx, const StepArgs &a, cudaStream_t st, bool with_ghosts, bool singly) {
  constexpr int V = StepVec<L, S>::value;
  if (V > 1 && !singly && !prefers_cells<L, S>(a) && vec_width<L, S>(a) == V)
    launch_vectors<L, S, V>(ctx, a, st, with_ghosts);
  else
    launch_vectors<L, S, 1>(ctx, a, st, with_ghosts);
}

template <class L, int S>
bool launch_step_boxes(ilbm_ctx *ctx, StepBoxes &p, cudaStream_t st) {
  constexpr int VV = StepVec<L, S>::value;
  int V = VV;
  int64_t total = 0;
  for (int n = 0; n < p.nbox; ++n) {
    V = std::min(V, vec_width<L, S>(p.a[n]));
    int64_t cells = 1;
    for (int d = 0; d < L::D; ++d) cells *= p.a[n].rhi[d] - p.a[n].rlo[d] + 1;
    total += cells;
  }
  if (total > kMaxLaunchCells) return false;
  uint32_t blocks = 0;
  for (int n = 0; n < p.nbox; ++n) {
    plan_vectors(p.a[n], L::D, V);
    p.a[n].ghost_blocks = 1;
    p.first[n] = blocks;
    blocks += plan_blocks(p.a[n], V);
  }
  p.first[p.nbox] = blocks;
  if (VV > 1 && V == VV)
    k_step_boxes<L, S, VV><<<blocks, kStepThreads, 0, st>>>(p);
  else
    k_step_boxes<L, S, 1><<<blocks, kStepThreads, 0, st>>>(p);
  ctx->launches++;
  return true;
}

template <class L, int S>
int launch_step_batch(ilbm_ctx *ctx, const StepArgs *d_args, const StepTile *d_tiles,
                             int ntiles, int V, int w, int blocks, const int *steps, const int *limit,
                             cudaStream_t st) {
  constexpr int VV = StepVec<L, S>::value;
  if (VV > 1 && V == VV)
    k_step_batch<L, S, VV><<<blocks, w, 0, st>>>(d_args, d_tiles, ntiles, steps, limit);
  else
    k_step_batch<L, S, 1><<<blocks, w, 0, st>>>(d_args, d_tiles, ntiles, steps, limit);
  ctx->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "batched level step launch");
  return ILBM_OK;
}

template <class L, int S>
int occupancy_step_batch(const ilbm_ctx *, int V, int w, int *per_sm) {
  constexpr int VV = StepVec<L, S>::value;
  cudaError_t e = (VV > 1 && V == VV)
                      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_step_batch<L, S, VV>, w, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_step_batch<L, S, 1>, w, 0);
  if (e != cudaSuccess) return cuda_fail(e, "batched level step occupancy");
  return ILBM_OK;
}

}  // namespace ilbm

// the launches of lattice Q in storage form S
#define ILBM_STEP_INSTANCE(Q, S)                                                                        \
  template int ilbm::vec_width<ilbm::Lat<Q>, S>(const ilbm::StepArgs &);                                \
  template void ilbm::launch_cells<ilbm::Lat<Q>, S>(ilbm_ctx *, const ilbm::StepArgs &, cudaStream_t,   \
                                                    bool, bool);                                              \
  template bool ilbm::launch_step_boxes<ilbm::Lat<Q>, S>(ilbm_ctx *, ilbm::StepBoxes &, cudaStream_t);  \
  template int ilbm::launch_step_batch<ilbm::Lat<Q>, S>(ilbm_ctx *, const ilbm::StepArgs *,             \
                                                        const ilbm::StepTile *, int, int, int, int,     \
                                                        const int *, const int *, cudaStream_t);        \
  template int ilbm::occupancy_step_batch<ilbm::Lat<Q>, S>(const ilbm_ctx *, int, int, int *);
