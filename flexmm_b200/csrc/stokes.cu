// Stokes FMM passes in FP64 (flexmm/kifmm2d/vector/stokes_fmm.py:550-858).
//
// A box carries 2 Neq + 1 values (row of np doubles): the equivalent forces
// (fx, fy) on Neq points of a circle plus one extra unknown of the corrected
// (pressure-augmented) forms; check values are the velocities (u, v) on Neq
// points plus the pressure at the circle's centre.  Per level:
//  * upward: partial = S2M (velocities on the check circle from the leaf's
//    sources; pressure row 0, as upwards_pass, stokes_fmm.py:259-291, ignores
//    kernel_add's pressure) + M2MC . children (extra unknowns excluded), then
//    the factored-SVD solve of the corrected equivalent-to-check form
//    (E2C_SVD, stokes_fmm.py:553-558);
//  * downward: partial locals += L2LC . parent local (real sibling groups) and
//    += M2L . source multipoles (the 40 offsets in one row-GEMM launch,
//    tiles of one parity class skipping absent offsets), then the C2E solve,
//    extra unknown dropped (stokes_fmm.py:712-733);
//  * evaluation: (u, v, p) from the leaf's local forces on the large circle
//    (local_expansion_evaluation, stokes_fmm.py:331-360) plus the colleagues'
//    sources (neighbor_evaluation, stokes_fmm.py:361-396).
// Solves and translations are FP64 tensor-core row GEMMs (rowgemm.cuh) on
// the plan's stream, gathers and scatters fused into their loads and stores.

#include <algorithm>

#include "dense.cuh"
#include "rowgemm.cuh"
#include "fmm.cuh"
#include "items.cuh"
#include "timing.cuh"

namespace fmmb {
namespace {

struct StokesCircles {
  const double *lx[FMM_MAX_LEVELS_DEV], *ly[FMM_MAX_LEVELS_DEV];  // large circle, per level
};

// Sums of Stokeslet (and stresslet) pairs at a target, unscaled (u, v times
// 1/(4 pi), p times 1/(2 pi) later).  With d = (dx, dy) = target - source,
// r2 = |d|^2 (kernel_apply_single, stokes_fmm.py:166-187):
//   u += -log(r2)/2 fx + dx s,  v += -log(r2)/2 fy + dy s,  p += s,
//   s = (d . f) / r2;
// a stresslet (kernel_apply_single_with_dipole, stokes_fmm.py:187-235) of
// strength sigma along the normal n adds, with c = 4 (d . n)(d . sigma) / r2^2,
//   u += c dx,  v += c dy,  p += c - 2 (n . sigma) / r2.
// The logarithms are summed as raw log2 values (lx, ly), from the passes'
// table, and the reciprocal is rcp_newton: about 24 FP64 instructions a pair
// where the library's logarithm and division took about 60 (a batch of 560k
// points, forward and adjoint: evaluation kernels 4.4 -> 1.9 ms, S2M 0.75 ->
// 0.45).
struct StokesSum {
  double lx = 0.0, ly = 0.0, u = 0.0, v = 0.0, p = 0.0;
  __device__ __forceinline__ void add(double dx, double dy, double fx, double fy, double l2, double i2) {
    const double s = fma(dx, fx, dy * fy) * i2;
    lx = fma(l2, fx, lx);
    ly = fma(l2, fy, ly);
    u = fma(dx, s, u);
    v = fma(dy, s, v);
    p += s;
  }
  __device__ __forceinline__ void add_dipole(double dx, double dy, double2 sg, double2 n, double i2) {
    const double c = 4.0 * fma(dx, n.x, dy * n.y) * i2 * (fma(dx, sg.x, dy * sg.y) * i2);
    u = fma(c, dx, u);
    v = fma(c, dy, v);
    p += fma(-2.0 * i2, fma(n.x, sg.x, n.y * sg.y), c);
  }
  static constexpr double kLog = -0.5 * 0.69314718055994530942;  // log2(r2) -> -log(r2)/2
};

// log2(r2) and 1 / r2 of a pair; false for a coincident pair when check is set
__device__ __forceinline__ bool stokes_radial(const LaplaceF64T &K, double r2, int check, double &l2,
                                              double &i2) {
  if (log2_rare_key(r2) < RCP_RARE) {
    l2 = K.at(r2);
    i2 = rcp_newton(r2);
    return true;
  }
  if (check && r2 == 0.0) return false;
  l2 = log2(r2);
  i2 = 1.0 / r2;
  return true;
}

// S2M: velocities at the large circle's points from the box's sources; one
// warp per S2M node, lane k owns check points k and k + 32.  DIP: the
// sources also carry stresslets (upwards_pass_dipole, stokes_fmm.py:294-322).
template <bool DIP>
__global__ void __launch_bounds__(128) k_stokes_s2m(int neq, int np, int L, StokesCircles cir,
                                                    const int *__restrict__ off,
                                                    const int *__restrict__ uplist,
                                                    const int *__restrict__ n_up_ptr,
                                                    const int *__restrict__ bot,
                                                    const int *__restrict__ top,
                                                    const double *__restrict__ xmid,
                                                    const double *__restrict__ ymid,
                                                    const double *__restrict__ sx,
                                                    const double *__restrict__ sy,
                                                    const double *__restrict__ fx,
                                                    const double *__restrict__ fy,
                                                    double *__restrict__ partial,
                                                    const double *__restrict__ sgx,
                                                    const double *__restrict__ sgy,
                                                    const double *__restrict__ dnx,
                                                    const double *__restrict__ dny) {
  __shared__ double qx[4][32], qy[4][32], qf[4][32], qg[4][32];
  __shared__ double2 qs[DIP ? 4 : 1][32], qn[DIP ? 4 : 1][32];
  __shared__ FunctorSmem<LaplaceF64T> fsm;
  LaplaceF64T K(KernelParams{});
  fsm.bind(K);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_up = *n_up_ptr;
  for (int i = blockIdx.x * 4 + warp; i < n_up; i += gridDim.x * 4) {
    const int g = uplist[i];
    const int m = node_level_of(off, L, g);
    const double cx = xmid[g], cy = ymid[g];
    double ex[2], ey[2];
    StokesSum sum[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = lane + 32 * h;
      ex[h] = k < neq ? cir.lx[m][k] : 0.0;
      ey[h] = k < neq ? cir.ly[m][k] : 0.0;
    }
    const int b = bot[g], e = top[g];
    for (int j0 = b; j0 < e; j0 += 32) {
      const int nj = min(32, e - j0);
      if (lane < nj) {
        qx[warp][lane] = sx[j0 + lane] - cx;
        qy[warp][lane] = sy[j0 + lane] - cy;
        qf[warp][lane] = fx[j0 + lane];
        qg[warp][lane] = fy[j0 + lane];
        if constexpr (DIP) {
          qs[warp][lane] = make_double2(sgx[j0 + lane], sgy[j0 + lane]);
          qn[warp][lane] = make_double2(dnx[j0 + lane], dny[j0 + lane]);
        }
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (lane + 32 * h < neq)
#pragma unroll 2
          for (int j = 0; j < nj; ++j) {
            const double dx = ex[h] - qx[warp][j], dy = ey[h] - qy[warp][j];
            double l2, i2;
            stokes_radial(K, fma(dy, dy, dx * dx), 0, l2, i2);
            sum[h].add(dx, dy, qf[warp][j], qg[warp][j], l2, i2);
            if constexpr (DIP) sum[h].add_dipole(dx, dy, qs[warp][j], qn[warp][j], i2);
          }
      __syncwarp();
    }
    const double us = 0.25 / M_PI;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = lane + 32 * h;
      if (k < neq) {
        partial[(size_t)g * np + k] = fma(StokesSum::kLog, sum[h].lx, sum[h].u) * us;
        partial[(size_t)g * np + neq + k] = fma(StokesSum::kLog, sum[h].ly, sum[h].v) * us;
      }
    }
  }
}

// Evaluation of an item (items.cuh): (u, v, p) rows of out (stride ld_out); the
// far field is the leaf's local forces on the large circle
// (local_expansion_evaluation, stokes_fmm.py:331-360), the near field its
// colleagues' sources, DIP with their stresslets (neighbor_evaluation(_dipole),
// stokes_fmm.py:361-441).
template <bool DIP>
struct StokesPolicy {
  using Kernel = LaplaceF64T;
  static constexpr int NOUT = 3, NV = 5;
  static constexpr int SMAX = DIP ? 384 : 512;  // 48 KB of static shared memory at most
  static constexpr bool kNear = true, kFar = true;
  struct Smem {
    double2 xy[SMAX], f[SMAX];
    double2 sg[DIP ? SMAX : 1], n[DIP ? SMAX : 1];
    double2 fxy[64], ff[64];  // the circle's points and forces
    double cx, cy;
    FunctorSmem<LaplaceF64T> fs;
  };
  template <int R>
  struct Tgt {};
  int neq, np, check;
  StokesCircles cir;
  const double *xmid, *ymid, *sx, *sy, *fx, *fy, *loc, *sgx, *sgy, *dnx, *dny;
  double *out;
  int64_t ld_out;

  __device__ __forceinline__ LaplaceF64T bind(Smem &sm) const {
    LaplaceF64T K(KernelParams{});
    sm.fs.bind(K);
    return K;
  }
  __device__ __forceinline__ void stage_far(Smem &sm, int g, int lev) const {
    const double *lf = loc + (size_t)g * np;
    for (int k = threadIdx.x; k < neq; k += EV_THREADS) {
      sm.fxy[k] = make_double2(cir.lx[lev][k], cir.ly[lev][k]);
      sm.ff[k] = make_double2(lf[k], lf[neq + k]);
    }
    if (threadIdx.x == 64) {
      sm.cx = xmid[g];
      sm.cy = ymid[g];
    }
  }
  __device__ __forceinline__ void stage(Smem &sm, int i, int j) const {
    sm.xy[i] = make_double2(sx[j], sy[j]);
    sm.f[i] = make_double2(fx[j], fy[j]);
    if constexpr (DIP) {
      sm.sg[i] = make_double2(sgx[j], sgy[j]);
      sm.n[i] = make_double2(dnx[j], dny[j]);
    }
  }
  template <class T>
  __device__ __forceinline__ void load_target(T &, int, const int *, int) const {}
  template <int R, bool D>
  __device__ __forceinline__ void pairs(const LaplaceF64T &K, const Smem &sm, const double2 *xy,
                                        const double2 *f, const double (&x)[R], const double (&y)[R],
                                        int lo, int hi, int G, int chk, double (&v)[R][NV]) const {
    StokesSum sum[R];
#pragma unroll
    for (int r = 0; r < R; ++r) sum[r] = {v[r][0], v[r][1], v[r][2], v[r][3], v[r][4]};
    auto one = [&](double dx, double dy, double2 q, int j, StokesSum &s, double l2, double i2) {
      s.add(dx, dy, q.x, q.y, l2, i2);
      if constexpr (D) s.add_dipole(dx, dy, sm.sg[j], sm.n[j], i2);
    };
    for (int j = lo; j < hi; j += G) {
      const double2 p = xy[j], q = f[j];
      double dx[R], dy[R], r2[R];
      unsigned key = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        dx[r] = x[r] - p.x;
        dy[r] = y[r] - p.y;
        r2[r] = fma(dy[r], dy[r], dx[r] * dx[r]);
        key = max(key, log2_rare_key(r2[r]));
      }
      if (key < RCP_RARE) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          one(dx[r], dy[r], q, j, sum[r], K.at(r2[r]), rcp_newton(r2[r]));
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          double l2, i2;
          // a pair is left out where it coincides, not where r2 underflows
          if (chk && dx[r] == 0.0 && dy[r] == 0.0) continue;
          stokes_radial(K, r2[r], 0, l2, i2);
          one(dx[r], dy[r], q, j, sum[r], l2, i2);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      v[r][0] = sum[r].lx;
      v[r][1] = sum[r].ly;
      v[r][2] = sum[r].u;
      v[r][3] = sum[r].v;
      v[r][4] = sum[r].p;
    }
  }
  template <int R>
  __device__ __forceinline__ void far_field(const LaplaceF64T &K, const Smem &sm, int, int,
                                            const double (&x)[R], const double (&y)[R], int warp,
                                            int sub, int G, double (&v)[R][NV]) const {
    double dx[R], dy[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dx[r] = x[r] - sm.cx;
      dy[r] = y[r] - sm.cy;
    }
    pairs<R, false>(K, sm, sm.fxy, sm.ff, dx, dy, (neq * warp) / EV_WARPS + sub,
                    (neq * (warp + 1)) / EV_WARPS, G, 0, v);
  }
  template <int R>
  __device__ __forceinline__ void sweep(const LaplaceF64T &K, const Smem &sm, const double (&x)[R],
                                        const double (&y)[R], const Tgt<R> &, int lo, int hi, int G,
                                        double (&v)[R][NV]) const {
    pairs<R, DIP>(K, sm, sm.xy, sm.f, x, y, lo, hi, G, check, v);
  }
  __device__ __forceinline__ void finish(const double (&v)[NV], double (&o)[NOUT]) const {
    o[0] = fma(StokesSum::kLog, v[0], v[2]) * (0.25 / M_PI);
    o[1] = fma(StokesSum::kLog, v[1], v[3]) * (0.25 / M_PI);
    o[2] = v[4] * (0.5 / M_PI);
  }
  __device__ __forceinline__ void store(int i, const double (&o)[NOUT]) const {
#pragma unroll
    for (int k = 0; k < NOUT; ++k) out[k * ld_out + i] = o[k];
  }
};

StokesCircles circles(const StokesArgs &a) {
  StokesCircles c{};
  for (int m = 0; m < a.th->L && m < FMM_MAX_LEVELS_DEV; ++m) {
    c.lx[m] = a.lev[m].lx;
    c.ly[m] = a.lev[m].ly;
  }
  return c;
}

// rows of x := ((b . U) . VHs), row-major np x np operators, n contiguous rows
void solve_rows(const StokesArgs &a, const double *u, const double *vhs, const double *b, double *x,
                double *tmp, int n, cudaStream_t s) {
  const int np = a.np;
  rowgemm(RowsContig{b, np, n, np}, StoreRows{tmp, np}, row_tiles(n), u, np, np, np, s);
  rowgemm(RowsContig{tmp, np, n, np}, StoreRows{x, np}, row_tiles(n), vhs, np, np, np, s);
}

}  // namespace

void run_stokes_upward(const StokesArgs &a, const double *fx, const double *fy, double *partial,
                       double *mult, cudaStream_t s) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  if (th.L < 3) return;
  FMMB_CHECK(th.L <= FMM_MAX_LEVELS_DEV, ERR_INVALID_ARGUMENT, "too many levels");
  const int np = a.np;
  PhaseTimer timer(PH_UPWARD, s);
  auto s2m = a.sgx ? k_stokes_s2m<true> : k_stokes_s2m<false>;
  s2m<<<work_grid(th.n_total(), 8), 128, 0, s>>>(a.neq, np, th.L, circles(a), td.dev_off.get(),
                                                 td.uplist.get(), td.n_up.get(), td.bot.get(),
                                                 td.top.get(), td.xmid.get(), td.ymid.get(),
                                                 td.sx.get(), td.sy.get(), fx, fy, partial, a.sgx,
                                                 a.sgy, a.dnx, a.dny);
  FMMB_CUDA(cudaGetLastError());
  int max_rows = 0;
  for (int m = 2; m < th.L; ++m) max_rows = std::max(max_rows, th.off[m + 1] - th.off[m]);
  DevBuf<double> tmp;
  tmp.alloc((size_t)max_rows * np, s);
  for (int m = th.L - 1; m >= 2; --m) {
    if (m <= th.L - 2) {  // partial of level m's parents = children . M2MC
      const int c_first = th.off[m + 1];
      const int n_groups = (th.off[m + 2] - th.off[m + 1]) / 4;
      if (n_groups > 0)
        rowgemm(RowsContig{mult + (size_t)c_first * np, 4 * (int64_t)np, n_groups, 4 * np},
                StoreParents{td.parent.get(), partial, c_first, np}, row_tiles(n_groups),
                a.lev[m].m2mc, np, np, 4 * np, s);
    }
    const int r0 = th.off[m], n = th.off[m + 1] - th.off[m];
    if (n > 0)
      solve_rows(a, a.lev[m].e2c_u, a.lev[m].e2c_vhs, partial + (size_t)r0 * np,
                 mult + (size_t)r0 * np, tmp.get(), n, s);
  }
}

void run_stokes_downward(const StokesArgs &a, const double *mult, double *ple, double *loc,
                         cudaStream_t s) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  if (th.L < 3) return;
  const int np = a.np;
  int max_groups = 0, max_rows = 0;
  for (int m = 2; m < th.L; ++m) {
    max_groups = std::max(max_groups, th.rg_hi[m] - th.rg_lo[m]);
    max_rows = std::max(max_rows, th.off[m + 1] - th.off[m]);
  }
  DevBuf<double> tmp;
  tmp.alloc((size_t)std::max(max_rows, 1) * np, s);
  for (int m = 2; m < th.L; ++m) {
    const int lo = th.rg_lo[m], n_groups = th.rg_hi[m] - th.rg_lo[m];
    if (n_groups > 0) {
      if (m >= 3) {  // L2L from level m-1 (stokes_fmm.py:726-733)
        PhaseTimer timer(PH_DOWNWARD, s);
        rowgemm(ParentRows{td.rg.get(), td.parent.get(), loc, lo, n_groups, np},
                AddChildRows{td.rg.get(), ple, lo, np}, row_tiles(n_groups), a.lev[m - 1].l2lc,
                4 * np, 4 * np, np, s);
      }
      // M2L: tiles of one parity class, absent offsets skipped
      PhaseTimer timer(PH_M2L, s);
      const int tpc = row_tiles(n_groups);
      rowgemm(M2LRows{td.rg.get(), td.il.get(), mult, lo, n_groups, np, tpc},
              AddGroupRows{td.rg.get(), ple, lo, np}, 4 * tpc, a.lev[m].m2l_cat, np, np, np, s);
    }
    const int r0 = th.off[m], nr = th.off[m + 1] - th.off[m];
    if (nr > 0)
      solve_rows(a, a.lev[m].c2e_u, a.lev[m].c2e_vhs, ple + (size_t)r0 * np, loc + (size_t)r0 * np,
                 tmp.get(), nr, s);
  }
}

void run_stokes_evaluate(const StokesArgs &a, const double *fx, const double *fy, const double *loc,
                         const double *txs, const double *tys, const uint64_t *tkeys,
                         const int *tperm, int64_t m, int check, double *out, int64_t ld_out,
                         cudaStream_t s) {
  if (m == 0) return;
  const TreeDev &td = *a.td;
  PassArgs pa{};
  pa.th = a.th;
  pa.td = a.td;
  EvalItems it;
  eval_items(pa, tkeys, m, it, s);
  PhaseTimer timer(PH_EVAL, s);
  const ItemArgs ia{it.items.get(), it.n_items.get(), it.n_items.get() + 1, td.coll.get(),
                    td.bot.get(),   td.top.get(),     txs,                 tys, tperm};
  auto launch = [&](auto pt, auto blocks) {
    using Pol = typename decltype(pt)::type;
    constexpr int B = decltype(blocks)::value;
    Pol pol{};
    pol.neq = a.neq;
    pol.np = a.np;
    pol.check = check;
    pol.cir = circles(a);
    pol.xmid = td.xmid.get();
    pol.ymid = td.ymid.get();
    pol.sx = td.sx.get();
    pol.sy = td.sy.get();
    pol.fx = fx;
    pol.fy = fy;
    pol.loc = loc;
    pol.sgx = a.sgx;
    pol.sgy = a.sgy;
    pol.dnx = a.dnx;
    pol.dny = a.dny;
    pol.out = out;
    pol.ld_out = ld_out;
    k_items<Pol, B><<<work_grid(a.th->n_total() + m / EVAL_CHUNK + 1, B), EV_THREADS, 0, s>>>(pol, ia);
  };
  if (a.sgx)
    launch(TypeOf<StokesPolicy<true>>{}, std::integral_constant<int, 4>{});
  else
    launch(TypeOf<StokesPolicy<false>>{}, std::integral_constant<int, 6>{});
  FMMB_CUDA(cudaGetLastError());
}

}  // namespace fmmb
