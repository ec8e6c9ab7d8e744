// The whole forcing chain of a small body in one launch (included by ib.cu).
//
// update_forcing of a body with a few hundred markers (IBMarkerDF.cpp:
// 1522-1917, one MDF iteration) is a chain of tiny stages: kinematics and
// interpolation, operator and solve, spreading, export.  As launches of their
// own (up to ten kernels and three memsets of 2-5 us, each waiting for the one
// before) they are bound by launch latency on the device and by API calls on
// the host.  Here one cluster of kChainCtas blocks runs them with a cluster
// barrier between stages.  Measured (B200, per step, with the stages' later
// changes): the 1024 x 512 FP32 cylinder (126 markers) 56 -> 36 us with its
// one-launch record; the pitching airfoil (240 markers, operator rebuilt) 115 ->
// 64 us; the finest level of the three-level cylinder (503 markers) 4 x 26 us of
// stages -> 4 x 21 us.  Eight blocks measured 51 us instead of 33 us cold on the
// last.  Which bodies take it: chain_markers (ib.cu).
//
// Stages:
//   1  a warp per marker: its position (moving bodies), kernel weights, the
//      velocity interpolated from rho, u formed on the spot at its stencil's
//      cells (so no band-wide macro pass), the right-hand side; the spread
//      force of its stencil's cells is zeroed; a warp per band row zeroes the
//      exported force
//   2  the marker forces: explicit; the stored inverse, a warp per row with the
//      right-hand side in shared memory; or CG with the operator built in
//      shared memory, each block holding the dense rows of its share of the
//      markers, z and p replicated, two cluster barriers per iteration
//   3  spreading (atomics; FP64 fixed bodies: the fixed-order gather)
//   4  export at the stencils' cells, rho formed on the spot; the marker sum
// The arithmetic of each stage is that of the separate kernels; FP64 storage
// keeps the reference's summation order in interpolation and spreading.

constexpr int kChainCtas = 16;       // non-portable cluster size: half of it doubled every stage
constexpr int kChainThreads = 512;

// dynamic shared memory of the chain for n markers.  CG: the block's rows of
// A, z and p of every marker, x, r, Ap, b and diagonal of its own rows, the
// reduction slots, the markers' weights and cells; stored inverse: the
// right-hand side
// a marker's weights in shared memory: an odd stride, so that consecutive
// markers' weights lie in different banks (stride 16 made every read of the
// operator's build a 32-way conflict: 77 -> 73 us of a 32-case batch step)
__host__ __device__ constexpr int chain_stride(int dim) { return 5 * dim + (dim == 2 ? 1 : 2); }
__host__ __device__ inline size_t chain_shared(int mode, int n, int dim, int ctas = kChainCtas) {
  const size_t rows = (size_t)(n + ctas - 1) / ctas;
  if (mode == 2)
    return (rows * n + 6 * (size_t)n + 13 * rows + 2 * (size_t)ctas * 6 + 8 + (chain_stride(dim) + 2) * (size_t)n) *
           sizeof(double);
  return mode == 1 ? 3 * (size_t)n * sizeof(double) : 0;
}

// interpolation of marker m by one warp (interp_one / interp_seq with the
// velocities formed at the stencil's cells); ORDERED: the reference's order;
// left: the status bit of a stencil that leaves the band
template <class L, int S, bool ORDERED>
__device__ __forceinline__ void chain_interp(const StepArgs &sa, const IBCase &k, const IBArgs &a, int m,
                                             int lane, int left) {
  const double px = k.xyz[m], py = k.xyz[m + a.n], pz = k.xyz[m + 2 * a.n];
  const double d = (a.dim == 3) ? X::mul(X::mul(a.dx[0], a.dx[1]), a.dx[2]) : X::mul(a.dx[0], a.dx[1]);
  int i0, j0, k0;
  double wx, wy, wz;
  if (k.sw) {  // markers that do not move: their weights once
    i0 = cell_of(px, a.plo[0], a.dx[0]);
    j0 = cell_of(py, a.plo[1], a.dx[1]);
    k0 = (a.dim == 3) ? cell_of(pz, a.plo[2], a.dx[2]) : 0;
    wx = k.sw[m].w[0][lane % 5];
    wy = k.sw[m].w[1][lane % 5];
    wz = k.sw[m].w[2][lane % 5];
  } else {
    marker_weights(a, px, py, pz, lane, i0, j0, k0, wx, wy, wz);
  }
  if (k.tw && lane < 5) {
    double *row = k.tw + (int64_t)kTabStride * m;
    row[lane] = wx;
    row[5 + lane] = wy;
    row[10 + lane] = wz;
  }
  if (k.tc && lane == 0) k.tc[m] = make_int4(i0, j0, k0, 0);
  const int ilo = a.dlo[0] - 2, ihi = a.dhi[0] + 2, jlo = a.dlo[1] - 2, jhi = a.dhi[1] + 2;
  const int klo = (a.dim == 3) ? a.dlo[2] - 2 : 0, khi = (a.dim == 3) ? a.dhi[2] + 2 : 0;
  constexpr int npts = (L::D == 3) ? 125 : 25;
  double s[4] = {0.0, 0.0, 0.0, 0.0};  // u, v, w, partition
#pragma unroll 1
  for (int it = 0; it < (npts + 31) / 32; ++it) {
    const int t = lane + 32 * it, tt = t < npts ? t : 0;
    const int ii = tt / (L::D == 3 ? 25 : 5), jj = (tt / (L::D == 3 ? 5 : 1)) % 5, kk = L::D == 3 ? tt % 5 : 2;
    const double tU = __shfl_sync(0xffffffffu, wx, ii), tV = __shfl_sync(0xffffffffu, wy, jj);
    const double tW = __shfl_sync(0xffffffffu, wz, kk);
    const int ip = i0 + ii - 2, jp = j0 + jj - 2, kp = (L::D == 3) ? k0 + kk - 2 : 0;
    const double dvl = (L::D == 3) ? X::mul(X::mul(tU, tV), tW) : X::mul(tU, tV);
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    if (t < npts && in_band(a, ip, jp, kp)) {  // (every cell the export visits starts from zero)
      const int64_t e = bidx(a, ip, jp, kp);
      k.EFI[e] = k.EFI[e + a.nb] = k.EFI[e + 2 * a.nb] = 0.0;
    }
    if (t < npts && dvl != 0.0 && ip >= ilo && ip <= ihi && jp >= jlo && jp <= jhi && kp >= klo && kp <= khi) {
      if (!in_band(a, ip, jp, kp)) {
        atomicOr(k.status, left);
      } else {
        double m4[4];
        band_macro_value<L, S>(sa, ip, jp, kp, m4);
        c[0] = X::mul(X::mul(dvl, m4[1]), d);
        c[1] = X::mul(X::mul(dvl, m4[2]), d);
        if (L::D == 3) c[2] = X::mul(X::mul(dvl, m4[3]), d);
        c[3] = X::mul(dvl, d);
      }
    }
    if constexpr (ORDERED) {
      // the points in the reference's order (i, then j, then k innermost):
      // lane order; every lane forms the same sums
      const int cnt = min(32, npts - 32 * it);
      for (int l = 0; l < cnt; ++l)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (e != 2 || L::D == 3) s[e] = X::add(s[e], __shfl_sync(0xffffffffu, c[e], l));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = X::add(s[e], c[e]);
    }
  }
  if constexpr (!ORDERED) {
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] = X::add(s[e], __shfl_xor_sync(0xffffffffu, s[e], o));
  }
  if (lane == 0) {
    if (a.renorm_interp && s[3] > 0.0)
      for (int e = 0; e < 3; ++e) s[e] = X::div(s[e], s[3]);
    double U[3] = {0.0, 0.0, 0.0};
    if (k.mode == 1) target_of(a, m, k.xyz, k.tgt, U[0], U[1], U[2]);
    for (int e = 0; e < 3; ++e) {
      k.uvw[m + e * a.n] = s[e];
      k.F[m + e * a.n] = 0.0;
      if (k.mode == 1) k.rhs[m + e * k.ld] = X::div(X::sub(U[e], s[e]), a.dt);
    }
  }
}

// row `row` of the stored inverse times the right-hand side b (3 x n), one warp
template <class TA>
__device__ __forceinline__ void chain_dense_row(const IBCase &k, const TA *Ainv, const double *b, int n, int row,
                                                int lane) {
  double s[3] = {0.0, 0.0, 0.0};
  const TA *Ar = Ainv + (size_t)row * k.ld;
  for (int h0 = lane; h0 < n; h0 += 256) {
    TA v[8];  // eight loads in flight
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = (h0 + 32 * u < n) ? Ar[h0 + 32 * u] : TA(0);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (h0 + 32 * u < n) {
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] += double(v[u]) * b[h0 + 32 * u + c * n];
      }
  }
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < 3; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
  if (lane == 0)
    for (int c = 0; c < 3; ++c) k.F[row + c * n] = s[c];
}

// Jacobi-preconditioned CG (ivc_cg_block's iteration) over the cluster: block
// `rank` owns rows [r0, r0 + nl) as dense rows of A in its shared memory, up to
// four consecutive ones per warp.  A product reads a column's p once for a
// warp's rows and skips the 32-column chunks none of them couples to (a marker
// couples within four cells, 60-100 of 384 columns): with a row at a time over
// all columns the loads of p from shared memory alone took 3,500 cycles per
// product of 48 rows.  Every block holds z and p of all markers; a block's z
// rows and partial sums go to all blocks through distributed shared memory, and
// each sums the partials in the same order, so all blocks take the same branches.
// The first writes into other blocks' shared memory (z, slot) follow the
// operator's build and need every block of the cluster to have started: the
// function arrives at the cluster's barrier before that build and waits after
// it, whatever its caller did before.
template <int CTAS>
__device__ __forceinline__ void chain_cg(cgrp::cluster_group &cl, const IBCase &k, const IBArgs &a, double *sh) {
  constexpr int NW = kChainThreads / 32, RW = 4;
  const int n = a.n, rank = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int rows = (n + CTAS - 1) / CTAS, r0 = min(n, rank * rows), nl = min(n, r0 + rows) - r0;
  int4 *tc = reinterpret_cast<int4 *>(sh);  // first: 16-byte aligned whatever n is
  const int ws = chain_stride(a.dim);
  double *tw = sh + 2 * (size_t)n, *A = tw + (size_t)ws * n, *z = A + (size_t)rows * n, *p = z + 3 * n;
  double *x = p + 3 * n, *r = x + 3 * rows, *ap = r + 3 * rows, *b = ap + 3 * rows, *dg = b + 3 * rows;
  double *slot = dg + rows;  // [2][CTAS][6]
  double *tot = slot + 2 * CTAS * 6;
  // the operator's entries over all blocks (rank 0's counts): beyond the capacity
  // that the sparse operator has, the body is refused as it is there
  __shared__ int entries;
  if (tid == 0) entries = 0;
  cl.barrier_arrive();  // (waited for before the first remote write)
  // the step's weight table, and the start: zero, the last solution, or the
  // extrapolation of the last two
#pragma unroll 4
  for (int t = tid; t < kTabStride * n; t += kChainThreads) {
    const double v = k.tw[t];
    if (t % kTabStride < 5 * a.dim) tw[t / kTabStride * ws + t % kTabStride] = v;
  }
  for (int t = tid; t < n; t += kChainThreads) tc[t] = k.tc[t];
  const int h = *k.hist, warm = h < 2 ? h : 2;
  for (int t = tid; t < 3 * n; t += kChainThreads)
    p[t] = !warm ? 0.0 : (warm == 1 ? k.X[t] : X::sub(X::mul(2.0, k.X[t]), k.Xh[t]));
  // this thread's entry of the block's vectors (3 nl <= the block's threads)
  const bool own = tid < 3 * nl;
  const int oc = own ? tid / nl : 0, oi = own ? tid - oc * nl : 0, og = r0 + oi + oc * n;
  if (own) {
    double U[3];
    target_of(a, r0 + oi, k.xyz, k.tgt, U[0], U[1], U[2]);
    b[tid] = X::div(X::sub(oc == 0 ? U[0] : (oc == 1 ? U[1] : U[2]), k.uvw[og]), a.dt);
  }
  __syncthreads();
  // the operator's rows
  const int rw = (nl + NW - 1) / NW, i0 = wid * rw, ni = max(0, min(nl - i0, rw));  // rw <= RW
  uint32_t chunks = 0;
  int coupled = 0;
  for (int j0 = 0; j0 < n; j0 += 32) {
    const int j = j0 + lane;
    bool any = false;
    for (int i = 0; i < ni; ++i) any = any || (j < n && may_couple_tab(a, tc, r0 + i0 + i, j));
    if (!__any_sync(0xffffffffu, any)) continue;
    chunks |= 1u << (j0 >> 5);
    if (j < n)
      for (int i = 0; i < ni; ++i) {
        const int row = r0 + i0 + i;
        const bool c = may_couple_tab(a, tc, row, j);
        const double v = c ? ivc_entry_tab(a, tw, tc, row, j, k.reg, ws) : 0.0;
        coupled += c;
        A[(size_t)(i0 + i) * n + j] = v;
        if (row == j) dg[i0 + i] = v;
      }
  }
  cl.barrier_wait();  // every block of the cluster runs
  for (int o = 16; o > 0; o >>= 1) coupled += __shfl_xor_sync(0xffffffffu, coupled, o);
  if (lane == 0 && coupled) atomicAdd(cl.map_shared_rank(&entries, 0), coupled);  // (read after the next barrier)
  __syncthreads();
  // ap = A p on the block's rows
  auto product = [&]() {
    double s[RW][3];
#pragma unroll
    for (int i = 0; i < RW; ++i) s[i][0] = s[i][1] = s[i][2] = 0.0;
    for (uint32_t m = chunks; m; m &= m - 1) {
      const int j = 32 * (__ffs(m) - 1) + lane;
      if (j >= n) continue;
      const double q0 = p[j], q1 = p[j + n], q2 = p[j + 2 * n];
#pragma unroll
      for (int i = 0; i < RW; ++i)
        if (i < ni) {
          const double v = A[(size_t)(i0 + i) * n + j];
          s[i][0] += v * q0;
          s[i][1] += v * q1;
          s[i][2] += v * q2;
        }
    }
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      if (i >= ni) continue;  // (the same for the whole warp)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) s[i][c] += __shfl_xor_sync(0xffffffffu, s[i][c], o);
      if (lane < 3) ap[i0 + i + lane * nl] = lane == 0 ? s[i][0] : (lane == 1 ? s[i][1] : s[i][2]);
    }
    __syncthreads();
  };
  int red = 0;  // selects the reduction slots
  // warp w < 6: the sum of f . g over the block's rows of component w % 3, sent
  // to every block; after the cluster barrier tot holds all blocks' sums
  auto send = [&](const double *f, const double *g) {
    const int c = wid % 3;
    double s = 0.0;
    for (int i = lane; i < nl; i += 32) s += f[i + c * nl] * g[i + c * nl];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < CTAS) cl.map_shared_rank(slot, lane)[(red * CTAS + rank) * 6 + wid] = s;
  };
  auto collect = [&](int count) {
    cl.sync();
    if (tid < count) {
      double s = 0.0;
      for (int q = 0; q < CTAS; ++q) s += slot[(red * CTAS + q) * 6 + tid];
      tot[tid] = s;
    }
    __syncthreads();
    red ^= 1;
  };
  // r = b - A x0, z = r / diag (kept in ap for the sums)
  if (own) x[tid] = p[og];
  product();
  double zz = 0.0;
  auto precondition = [&](double rr) {
    zz = rr / dg[oi];
    r[tid] = rr;
    ap[tid] = zz;
    for (int q = 0; q < CTAS; ++q) cl.map_shared_rank(z, q)[og] = zz;
  };
  if (own) precondition(b[tid] - ap[tid]);
  __syncthreads();
  if (wid < 3) send(r, ap);
  else if (wid < 6) send(b, b);
  collect(6);
  double rz[3], bn[3];
  for (int c = 0; c < 3; ++c) {
    rz[c] = tot[c];
    bn[c] = sqrt(tot[3 + c]);
  }
  for (int t = tid; t < 3 * n; t += kChainThreads) p[t] = z[t];
  __syncthreads();
  bool done = false;
  int it = 0;
  for (; it < 500; ++it) {
    product();
    if (own) b[tid] = p[og];  // (b is needed no longer: the block's rows of p)
    __syncthreads();
    if (wid < 3) send(b, ap);
    collect(3);
    if (own) {
      const double t = tot[oc], al = (t != 0.0) ? (oc == 0 ? rz[0] : (oc == 1 ? rz[1] : rz[2])) / t : 0.0;
      x[tid] += al * p[og];
      precondition(r[tid] - al * ap[tid]);
    }
    __syncthreads();
    if (wid < 3) send(r, ap);
    else if (wid < 6) send(r, r);
    collect(6);
    bool ok = true;
    double beta[3];
    for (int c = 0; c < 3; ++c) {
      beta[c] = (rz[c] != 0.0) ? tot[c] / rz[c] : 0.0;
      rz[c] = tot[c];
      ok = ok && (sqrt(tot[3 + c]) <= k.cg_tol * bn[c]);
    }
    if (ok) {
      done = true;
      ++it;
      break;
    }
    for (int j = tid; j < n; j += kChainThreads)
#pragma unroll
      for (int c = 0; c < 3; ++c) p[j + c * n] = z[j + c * n] + beta[c] * p[j + c * n];
    __syncthreads();
  }
  // every block has read X, Xh and hist before its first cluster barrier
  if (rank == 0 && tid == 0) {
    *k.iters = it;
    if (!done) atomicOr(k.status, 4);
    if (entries > k.nnz_cap) atomicOr(k.status, 2);
    *k.hist = (h + 1 < 2) ? h + 1 : 2;
  }
  if (own) {
    if (warm) k.Xh[og] = k.X[og];
    k.X[og] = x[tid];
    k.F[og] = x[tid];
  }
}

template <class L, int S>
__device__ __forceinline__ void chain_body(const StepArgs &sa, const IBCase &k, double kc, double ks, double om,
                                           double *sh) {
  using R = typename Store<S>::R;
  constexpr bool ORDERED = S == ILBM_STORAGE_F64;
  cgrp::cluster_group cl = cgrp::this_cluster();
  const IBArgs &a = k.a;
  const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31;
  const int gt = rank * kChainThreads + tid, gsz = kChainCtas * kChainThreads;
  const int gw = gt >> 5, nw = gsz >> 5;
  const int n = a.n;
  // 1: markers and interpolation; the spread force starts from zero
  if (gt == 0) {
    k.fsum[0] = k.fsum[1] = k.fsum[2] = 0.0;
    k.status[0] = 0;
  }
  cl.sync();  // (the status is cleared before a stage may raise it)
  R *F = static_cast<R *>(const_cast<void *>(sa.force));
  const int i0 = max(a.blo[0], a.dlo[0]), i1 = min(a.blo[0] + a.bn[0] - 1, a.dhi[0]);
  for (int row = gw; row < a.bn[1] * a.bn[2]; row += nw) {
    const int j = a.blo[1] + row % a.bn[1], q = a.blo[2] + row / a.bn[1];
    if (k.periodic_band)  // (images are read outside the stencils)
      for (int i = lane; i < a.bn[0]; i += 32)
        for (int c = 0; c < 3; ++c) k.EFI[(int64_t)row * a.bn[0] + i + c * a.nb] = 0.0;
    if (j < a.dlo[1] || j > a.dhi[1] || (a.dim == 3 && (q < a.dlo[2] || q > a.dhi[2]))) continue;
    const int64_t m0 = midx(sa, i0, j, a.dim == 3 ? q : 0);
    for (int i = lane; i <= i1 - i0; i += 32)
      for (int c = 0; c < a.dim; ++c) F[m0 + i + c * sa.ms2] = R(0);
  }
  if (k.periodic_band) cl.sync();
  for (int m = gw; m < n; m += nw) {
    if (lane == 0 && k.moving) markers_one(a, kc, ks, om, m, k.xyz, k.ref, k.tgt, k.uvw, k.F);
    __syncwarp();
    chain_interp<L, S, ORDERED>(sa, k, a, m, lane, 1);
  }
  cl.sync();
  // 2: marker forces
  if (k.mode == 2) {
    chain_cg<kChainCtas>(cl, k, a, sh);
  } else if (k.mode == 1) {
    for (int t = tid; t < 3 * n; t += kChainThreads) sh[t] = k.rhs[t % n + (t / n) * k.ld];
    __syncthreads();
    for (int m = gw; m < n; m += nw) {
      if (k.Ainv32)
        chain_dense_row(k, k.Ainv32, sh, n, m, lane);
      else
        chain_dense_row(k, k.Ainv, sh, n, m, lane);
    }
  } else {
    for (int m = gt; m < n; m += gsz) force_explicit_one(a, m, k.xyz, k.tgt, k.uvw, k.F);
  }
  cl.sync();
  // 3: spreading
  if (ORDERED && k.gcells > 0) {
    for (int r = gt; r < k.gcells; r += gsz) {
      double ax, ay, az;
      gather_row(a, k.sw, k.F, k.growptr, k.gent, r, ax, ay, az);
      const int64_t t = k.gcell[r];
      k.EFI[t] = ax;
      k.EFI[t + a.nb] = ay;
      if (a.dim == 3) k.EFI[t + 2 * a.nb] = az;
    }
  } else {
    for (int m = gw; m < n; m += nw) {
      if (k.tc)
        spread_one_tab(a, m, lane, k.tw, k.tc, k.F, k.EFI, k.status);
      else
        spread_one(a, m, lane, k.xyz, k.F, k.EFI, k.status);
    }
  }
  cl.sync();
  if (k.periodic_band) {
    for (int t = gt; t < (int)a.nb; t += gsz) sum_boundary_cell(a, k.EFI, t);
    cl.sync();
  }
  // 4: export at the cells a force was spread to; the marker sum
  auto export_at = [&](int64_t t) {
    const double f[3] = {k.EFI[t], k.EFI[t + a.nb], a.dim == 3 ? k.EFI[t + 2 * a.nb] : 0.0};
    const int u = (int)t, i = a.blo[0] + u % a.bn[0], r = u / a.bn[0];
    const int j = a.blo[1] + r % a.bn[1], q = a.dim == 3 ? a.blo[2] + r / a.bn[1] : 0;
    if (i < a.dlo[0] || i > a.dhi[0] || j < a.dlo[1] || j > a.dhi[1] ||
        (a.dim == 3 && (q < a.dlo[2] || q > a.dhi[2])) || (f[0] == 0.0 && f[1] == 0.0 && f[2] == 0.0))
      return;
    double m4[4];
    band_macro_value<L, S>(sa, i, j, q, m4);
    const double dr = X::mul(a.dt, m4[0]);
    const int64_t m = midx(sa, i, j, q);
    F[m] = R(X::mul(dr, f[0]));
    F[m + sa.ms2] = R(X::mul(dr, f[1]));
    if (a.dim == 3) F[m + 2 * sa.ms2] = R(X::mul(dr, f[2]));
  };
  if (k.periodic_band) {
    for (int t = gt; t < (int)a.nb; t += gsz) export_at(t);
  } else if (k.gcells > 0) {
    for (int r = gt; r < k.gcells; r += gsz) export_at(k.gcell[r]);
  } else {
    // a warp per marker (cells shared by stencils are written with the same values)
    for (int m = gw; m < n; m += nw) {
      const int ci = cell_of(k.xyz[m], a.plo[0], a.dx[0]), cj = cell_of(k.xyz[m + n], a.plo[1], a.dx[1]);
      const int ck = a.dim == 3 ? cell_of(k.xyz[m + 2 * n], a.plo[2], a.dx[2]) : 0;
      for (int t = lane; t < (L::D == 3 ? 125 : 25); t += 32) {
        const int ip = ci + t / (L::D == 3 ? 25 : 5) - 2, jp = cj + (t / (L::D == 3 ? 5 : 1)) % 5 - 2;
        const int kp = L::D == 3 ? ck + t % 5 - 2 : 0;
        if (in_band(a, ip, jp, kp)) export_at(bidx(a, ip, jp, kp));
      }
    }
  }
  if (rank == kChainCtas - 1) marker_sum_block(a, k.F, k.fsum);
}

struct ChainArgs {
  StepArgs s;
  IBCase k;
};

template <class L, int S>
__global__ void __cluster_dims__(kChainCtas, 1, 1) __launch_bounds__(kChainThreads, 1)
    k_ib_chain(const __grid_constant__ ChainArgs c) {
  extern __shared__ __align__(16) double sh[];
  chain_body<L, S>(c.s, c.k, c.k.a.kc, c.k.a.ks, c.k.a.komega, sh);
}

// ---------------------------------------------------------------------------
// The batch's stages on the same functions.
// ---------------------------------------------------------------------------
// kinematics and interpolation, a warp per marker, with rho and u formed at the
// stencils' cells (a macro pass over every band cell of the batch and a marker
// kernel before it took 26 of 382 us per step on 32 cases); the spread force is
// zero on entry (k_b_export leaves it so).  The step's status starts here, in the
// launch that may already raise its first bit: a stencil outside the band
// raises kLeftBand, which k_b_record turns into status bit 1 at the step's end.
constexpr int kLeftBand = 32;
template <class L, int S>
__global__ void __launch_bounds__(128) k_b_interp(const IBCase *cs, const StepArgs *args, const ItemRef *list,
                                                  int64_t cnt, const int *steps, const int *limit) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < cnt; w += nw) {
    const ItemRef e = list[w];
    if (!live(steps, limit, e.c)) continue;
    const IBCase &k = cs[e.c];
    const int m = e.u;
    if (lane == 0) {
      if (m == 0) {
        k.fsum[0] = k.fsum[1] = k.fsum[2] = 0.0;
        atomicAnd(k.status, kLeftBand);  // (other warps may be raising this step's already)
      }
      if (k.moving) {
        int s = steps[e.c];
        if (s >= k.kin_steps) {
          if (m == 0) atomicOr(k.status, 16);  // ran past its kinematics table
          s = k.kin_steps - 1;
        }
        markers_one(k.a, k.kin[4 * s + 1], k.kin[4 * s + 2], k.kin[4 * s], m, k.xyz, k.ref, k.tgt, k.uvw, k.F);
      }
    }
    __syncwarp();
    chain_interp<L, S, false>(args[e.c], k, k.a, m, lane, kLeftBand);
  }
}

// the moving bodies' operator build and CG, a cluster per body (count, scan and
// fill of a CSR operator and a one-block CG on it took 101 us for the 16
// bodies of a 32-case batch; this takes 60 us, and its one launch leaves the
// stored-inverse solves beside it undisturbed: 382 -> 333 us per batch step with
// the interpolation above)
constexpr int kBatchCgCtas = 8;
__global__ void __cluster_dims__(kBatchCgCtas, 1, 1) __launch_bounds__(kChainThreads, 1)
    k_b_cluster_cg(const IBCase *cs, const int *list, const int *steps, const int *limit) {
  extern __shared__ __align__(16) double sh[];
  __shared__ IBCase k;  // (not through the global table: its fields are read all through the solve)
  const int c = list[blockIdx.x / kBatchCgCtas];
  if (!live(steps, limit, c)) return;  // the same for the whole cluster
  cgrp::cluster_group cl = cgrp::this_cluster();
  for (int w = threadIdx.x; w < (int)(sizeof(IBCase) / sizeof(int)); w += blockDim.x)
    reinterpret_cast<int *>(&k)[w] = reinterpret_cast<const int *>(cs + c)[w];
  __syncthreads();
  chain_cg<kBatchCgCtas>(cl, k, k.a, sh);
  cl.sync();  // no block leaves while another may still write to it
}
