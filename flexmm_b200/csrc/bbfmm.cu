// Black-box (Chebyshev) FMM passes in FP64 (flexmm/flexmm2d/bbfmm.py).
//
// The expansions of a box are p x p Chebyshev coefficients on the box scaled
// to [-1, 1]^2 (NQ = p^2, rows padded to np):
//  * S2M: Chebyshev moments of the box's sources,
//    M[a p + b] = sum_j T_a(x_j) T_b(y_j) tau_j (anterpolate2, bbfmm.py:11-24,
//    source2pMs, bbfmm.py:186-196); no check-to-equivalent step;
//  * M2M / L2L: the level-independent M2MC [NQ x 4NQ] and its transpose
//    (bbfmm.py:145-161) on the contiguous child rows of each parent group.  A
//    child's block of M2MC is the tensor product X (x) Y of two p x p matrices:
//    a row as a p x p matrix C goes to X C Y^T, 4 p^3 operations a child instead
//    of 2 p^4 (k_bb_shift).  Operators that are no such product (the entry point
//    takes any) go through the row GEMM;
//  * M2L: per level and offset VI K VI^T (bbfmm.py:101-122).  A width's 40
//    operators share a space of at most 64 columns for the smooth kernels
//    (fmm_bb_ops_set_basis): multipoles go into that basis, the KIFMM's M2L
//    kernel translates rows of 64 there, all levels in one launch, and the
//    results come back, a sixteenth of the work at p = 16.  Levels without
//    such a basis apply their operators in a row-GEMM launch
//    (rowgemm.cuh) over the stacked operators, each tile of 64 target boxes
//    of one parity class skipping the offsets absent for the whole tile;
//  * L2T: the local coefficients evaluated as a 2-D Chebyshev series
//    (chebeval2d1, bbfmm.py:25-31, L2targets, bbfmm.py:198-210);
//  * P2P: the same colleague sweep as the KIFMM evaluation.
// M2M, L2L and M2L are FP64 tensor-core row GEMMs (rowgemm.cuh) with their
// gathers and scatters fused into the loads and stores; moments and
// evaluation are the kernels below.

#include <algorithm>
#include <string>

#include "dense.cuh"
#include "rowgemm.cuh"
#include "fmm.cuh"
#include "sweep.cuh"
#include "timing.cuh"

namespace fmmb {
namespace {

constexpr int BB_MAX_P = 16;

// 2 / width per level: maps a box to [-1, 1]^2 (width_adj, bbfmm.py:122)
struct BBScale {
  double inv_hw[FMM_MAX_LEVELS_DEV];
};

// S2M moments, one warp per S2M node; lane owns outputs q = lane + 32 k
__global__ void __launch_bounds__(128) k_bb_s2m(int p, int np, int L, BBScale sc,
                                                const int *__restrict__ off,
                                                const int *__restrict__ uplist,
                                                const int *__restrict__ n_up_ptr,
                                                const int *__restrict__ bot,
                                                const int *__restrict__ top,
                                                const double *__restrict__ xmid,
                                                const double *__restrict__ ymid,
                                                const double *__restrict__ sx,
                                                const double *__restrict__ sy,
                                                const double *__restrict__ tau,
                                                double *__restrict__ mult) {
  __shared__ double Tx[4][32][BB_MAX_P], Ty[4][32][BB_MAX_P], tw[4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_up = *n_up_ptr, nq = p * p;
  int qa[8], qb[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int q = lane + 32 * k;
    qa[k] = q < nq ? q / p : 0;
    qb[k] = q < nq ? q % p : 0;
  }
  for (int i = blockIdx.x * 4 + warp; i < n_up; i += gridDim.x * 4) {
    const int g = uplist[i];
    const double a = sc.inv_hw[node_level_of(off, L, g)];
    const double cx = xmid[g], cy = ymid[g];
    const int b = bot[g], e = top[g];
    double acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.0;
    for (int j0 = b; j0 < e; j0 += 32) {
      const int nj = min(32, e - j0);
      if (lane < nj) {
        const double x = (sx[j0 + lane] - cx) * a, y = (sy[j0 + lane] - cy) * a;
        double t0 = 1.0, t1 = x, u0 = 1.0, u1 = y;
        Tx[warp][lane][0] = 1.0;
        Ty[warp][lane][0] = 1.0;
        for (int n = 1; n < p; ++n) {
          Tx[warp][lane][n] = t1;
          Ty[warp][lane][n] = u1;
          const double t2 = 2.0 * x * t1 - t0, u2 = 2.0 * y * u1 - u0;
          t0 = t1;
          t1 = t2;
          u0 = u1;
          u1 = u2;
        }
        tw[warp][lane] = tau[j0 + lane];
      }
      __syncwarp();
      for (int jj = 0; jj < nj; ++jj) {
        const double t = tw[warp][jj];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (lane + 32 * k < nq) acc[k] = fma(Tx[warp][jj][qa[k]] * Ty[warp][jj][qb[k]], t, acc[k]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int q = lane + 32 * k;
      if (q < np) mult[(size_t)g * np + q] = q < nq ? acc[k] : 0.0;
    }
  }
}

// Evaluation of an item (items.cuh): L2T as a 2-D Chebyshev series of the
// leaf's local coefficients, sum_a T_a(x) sum_b c[a p + b] T_b(y), the rows a
// split over the warps and the lanes of a target; P2P as in the KIFMM.
// NOUT = 3 adds the gradient in the target position: the series' derivative
// (T_n' by its recurrence, chebeval2d_dx / _dy, bbfmm.py:32-45) and the
// kernel's gradient.  500k sources, 250k targets, p = 16: potentials 0.85 ->
// 0.27 ms, the two gradient evaluations 2.55 -> 1.14 ms.
template <class KF, int NOUT>
struct BBPolicy : ChargePolicy<KF, NOUT, false, false> {
  using Base = ChargePolicy<KF, NOUT, false, false>;
  static constexpr bool kNear = true, kFar = true;
  using Smem = typename Base::Smem;
  int p, np;
  BBScale sc;
  const double *xmid, *ymid, *loc;

  __device__ __forceinline__ void stage_far(Smem &, int, int) const {}
  template <int R>
  __device__ __forceinline__ void far_field(const KF &, const Smem &, int g, int lev,
                                            const double (&x)[R], const double (&y)[R], int warp,
                                            int sub, int G, double (&v)[R][Base::NV]) const {
    const double a = sc.inv_hw[lev], cx = xmid[g], cy = ymid[g];
    const double *cr = loc + (size_t)g * np;
    // raw sums of a table functor are scaled at the end: divide that out here
    double su = 1.0, sg = a;  // d/dx = (2 / w) d/dxh
    if constexpr (KF::kLogTable) {
      su = 1.0 / KF::kFold;
      sg = a / KF::grad_fold(this->kp);
    }
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
      const double xh = ((r == 0 ? x[0] : x[R - 1]) - cx) * a;
      const double yh = ((r == 0 ? y[0] : y[R - 1]) - cy) * a;
      double ty[BB_MAX_P], dty[NOUT == 3 ? BB_MAX_P : 1];
      ty[0] = 1.0;
      ty[1] = yh;
      if (NOUT == 3) {
        dty[0] = 0.0;
        dty[NOUT == 3 ? 1 : 0] = 1.0;
      }
#pragma unroll
      for (int b = 2; b < BB_MAX_P; ++b) {
        ty[b] = 2.0 * yh * ty[b - 1] - ty[b - 2];
        if constexpr (NOUT == 3) dty[b] = 2.0 * ty[b - 1] + 2.0 * yh * dty[b - 1] - dty[b - 2];
      }
      double u = 0.0, gx = 0.0, gy = 0.0;
      double tp = 1.0, tc = xh;     // T_{ar-1}, T_ar as ar advances
      double dtp = 0.0, dtc = 1.0;  // their derivatives
      for (int ar = 0; ar < p; ++ar) {
        const double tx = ar == 0 ? 1.0 : tc, dtx = ar == 0 ? 0.0 : dtc;
        if ((ar & (EV_WARPS - 1)) == warp && ((ar / EV_WARPS) & (G - 1)) == sub) {
          double s = 0.0, sd = 0.0;
#pragma unroll
          for (int b = 0; b < BB_MAX_P; ++b)
            if (b < p) {
              const double c = __ldg(cr + ar * p + b);
              s = fma(c, ty[b], s);
              if constexpr (NOUT == 3) sd = fma(c, dty[b], sd);
            }
          u = fma(tx, s, u);
          if (NOUT == 3) {
            gx = fma(dtx, s, gx);
            gy = fma(tx, sd, gy);
          }
        }
        if (ar >= 1) {
          const double tn = 2.0 * xh * tc - tp;
          if (NOUT == 3) {
            const double dtn = 2.0 * tc + 2.0 * xh * dtc - dtp;
            dtp = dtc;
            dtc = dtn;
          }
          tp = tc;
          tc = tn;
        }
      }
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (k == r) {
          if constexpr (NOUT == 1) {
            v[k][0] += u;
          } else {
            v[k][0] += u * su;
            v[k][1] += gx * sg;
            v[k][2] += gy * sg;
          }
        }
    }
  }
};

// M2M (UP: the children's rows into their parent's, overwritten) or L2L (the
// parent's row added to the children's) of one level by the operators' tensor
// factors, a warp a parent or a child.  With D = X C Y^T as D^T = (Y C^T) X^T
// the first product's accumulators are the second's operand as they lie (the k
// index of a DMMA is free: 2 q and 2 q + 1 of the two steps), C is read from
// global memory in the operand's own layout, and only the factors (fragments,
// sep: Y then X, bb_shift_fragments in capi.cu) are staged.  Bound by latency
// and the launches on coarse levels.  500k sources, p = 16, three passes of five
// levels: M2M 1051 -> 176 us, L2L 477 -> 214 us (row GEMMs before).
constexpr int SHIFT_WARPS = 4;
template <int P, bool UP>
__global__ void __launch_bounds__(32 * SHIFT_WARPS)
    k_bb_shift(int p, int np, const double *__restrict__ sep, const int *__restrict__ parent,
               const int *__restrict__ rg, int first, int units, double *rows) {
  constexpr int NB = P / 8, KS = P / 4, F = 4 * P * P;
  __shared__ double fy[F], fx[F];
  for (int i = threadIdx.x; i < F; i += 32 * SHIFT_WARPS) {
    fy[i] = __ldg(sep + i);
    fx[i] = __ldg(sep + F + i);
  }
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  for (int u = blockIdx.x * SHIFT_WARPS + warp; u < units; u += gridDim.x * SHIFT_WARPS) {
    double out[NB][NB][2];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) out[i][j][0] = out[i][j][1] = 0.0;
    auto load = [&](const double *row, double (&b)[NB][KS]) {
#pragma unroll
      for (int cb = 0; cb < NB; ++cb)
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
          b[cb][ks] = 8 * cb + g < p && 4 * ks + q < p ? row[(8 * cb + g) * p + 4 * ks + q] : 0.0;
    };
    auto shift = [&](int c, const double (&b)[NB][KS]) {
#pragma unroll
      for (int rb = 0; rb < NB; ++rb) {
        double v[NB][2];
#pragma unroll
        for (int cb = 0; cb < NB; ++cb) {
          v[cb][0] = v[cb][1] = 0.0;
#pragma unroll
          for (int ks = 0; ks < KS; ++ks)
            dmma(v[cb], fy[((c * NB + rb) * KS + ks) * 32 + lane], b[cb][ks]);
        }
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int cb = 0; cb < NB; ++cb)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              dmma(out[rb][nb], v[cb][h], fx[(((c * NB + nb) * NB + cb) * 2 + h) * 32 + lane]);
      }
    };
    double *dst;
    if (UP) {
      const double *src = rows + (size_t)(first + 4 * u) * np;
      dst = rows + (size_t)parent[first + 4 * u] * np;
      double b[4][NB][KS];
#pragma unroll
      for (int c = 0; c < 4; ++c) load(src + (size_t)c * np, b[c]);
#pragma unroll
      for (int c = 0; c < 4; ++c) shift(c, b[c]);
    } else {
      const int node = rg[first + (u >> 2)] + (u & 3);
      dst = rows + (size_t)node * np;
      double b[NB][KS];
      load(rows + (size_t)parent[node] * np, b);
      shift(u & 3, b);
    }
#pragma unroll
    for (int rb = 0; rb < NB; ++rb)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int a = 8 * nb + 2 * q + j, b = 8 * rb + g;
          if (a < p && b < p) dst[a * p + b] = UP ? out[rb][nb][j] : dst[a * p + b] + out[rb][nb][j];
        }
  }
}

template <bool UP>
void bb_shift(const BBArgs &b, int first, int units, double *rows, cudaStream_t s) {
  const dim3 grid(work_grid((units + SHIFT_WARPS - 1) / SHIFT_WARPS, 4));
  launch_pdl(b.p <= 8 ? k_bb_shift<8, UP> : k_bb_shift<16, UP>, grid, dim3(32 * SHIFT_WARPS), 0, s,
             b.p, b.np, UP ? b.m2m_sep : b.l2l_sep, b.td->parent.get(), b.td->rg.get(), first, units,
             rows);
}

BBScale bb_scale(const TreeHost &th) {
  BBScale sc{};
  for (int m = 0; m < th.L && m < FMM_MAX_LEVELS_DEV; ++m) sc.inv_hw[m] = 2.0 / th.width[m];
  return sc;
}

}  // namespace

void run_bb_upward(const BBArgs &b, const double *tau_s, double *mult, cudaStream_t s) {
  const TreeHost &th = *b.th;
  const TreeDev &td = *b.td;
  if (th.L < 3) return;
  FMMB_CHECK(th.L <= FMM_MAX_LEVELS_DEV, ERR_INVALID_ARGUMENT, "too many levels");
  const int np = b.np;
  const BBScale sc = bb_scale(th);
  PhaseTimer timer(PH_UPWARD, s);
  k_bb_s2m<<<work_grid(th.n_total(), 8), 128, 0, s>>>(b.p, np, th.L, sc, td.dev_off.get(), td.uplist.get(),
                                   td.n_up.get(), td.bot.get(), td.top.get(), td.xmid.get(),
                                   td.ymid.get(), td.sx.get(), td.sy.get(), tau_s, mult);
  FMMB_CUDA(cudaGetLastError());
  for (int m = th.L - 2; m >= 2; --m) {
    const int c_first = th.off[m + 1];
    const int n_groups = (th.off[m + 2] - th.off[m + 1]) / 4;
    if (n_groups == 0) continue;
    if (b.m2m_sep) {
      bb_shift<true>(b, c_first, n_groups, mult, s);
      continue;
    }
    // parent rows = children rows (contiguous, 4np wide) . M2MC^T (fmm.py:93-96)
    rowgemm(RowsContig{mult + (size_t)c_first * np, 4 * (int64_t)np, n_groups, 4 * np},
            StoreParents{td.parent.get(), mult, c_first, np}, row_tiles(n_groups), b.m2mct, np, np,
            4 * np, s);
  }
}

void run_bb_downward(const BBArgs &b, const double *mult, double *ple, double *z, double *zl,
                     cudaStream_t s) {
  const TreeHost &th = *b.th;
  const TreeDev &td = *b.td;
  if (th.L < 3) return;
  const int np = b.np;
  static_assert(BB_RANK <= 64, "the KIFMM's M2L takes rows of at most 64");
  if (b.any_fast) {
    // M2L of these levels in one launch of the KIFMM's kernel, on rows of at most
    // 64: the coefficients themselves (p <= 8), or those in the common basis
    const bool basis = np > BB_RANK;
    // into the basis and back, all these levels in one launch each
    RowsLevels in{}, back{};
    for (int m = 2; basis && m < th.L; ++m)
      if (b.fast[m]) {
        in.add(th.off[m], th.off[m + 1] - th.off[m], b.q[m]);
        back.add(th.off[m], th.off[m + 1] - th.off[m], b.q[m] + (size_t)np * BB_RANK);
      }
    in.base = mult;
    in.ld = np;
    back.base = zl;
    back.ld = BB_RANK;
    if (basis)
      rowgemm(in, StoreRows{z, BB_RANK}, in.tile0[in.n], b.q[2], BB_RANK, BB_RANK, np, s);
    PassArgs a{};
    a.np = basis ? BB_RANK : np;
    a.th = b.th;
    a.td = b.td;
    a.ops_dev = b.ops_dev;
    run_m2l(a, basis ? z : mult, basis ? zl : ple, s);
    if (basis) rowgemm(back, StoreRows{ple, np}, back.tile0[back.n], b.q[2], np, np, BB_RANK, s);
  }
  for (int m = 2; m < th.L; ++m) {
    const int lo = th.rg_lo[m], n_groups = th.rg_hi[m] - th.rg_lo[m];
    if (n_groups == 0) continue;
    if (m >= 3) {  // L2L from level m-1: children += parent local . M2MC (bbfmm.py:161, fmm.py:140-147)
      PhaseTimer timer(PH_DOWNWARD, s);
      if (b.l2l_sep)
        bb_shift<false>(b, lo, 4 * n_groups, ple, s);
      else
        rowgemm(ParentRows{td.rg.get(), td.parent.get(), ple, lo, n_groups, np},
                AddChildRows{td.rg.get(), ple, lo, np}, row_tiles(n_groups), b.m2mc, 4 * np,
                4 * np, np, s);
    }
    if (!b.fast[m]) {  // M2L of level m: tiles of one parity class, absent offsets skipped (fmm.py:118-131)
      PhaseTimer timer(PH_M2L, s);
      const int tpc = row_tiles(n_groups);
      rowgemm(M2LRows{td.rg.get(), td.il.get(), mult, lo, n_groups, np, tpc},
              AddGroupRows{td.rg.get(), ple, lo, np}, 4 * tpc, b.m2l_cat[m], np, np, np, s);
    }
  }
}

void run_bb_evaluate(const BBArgs &b, const double *tau_s, const double *loc, const double *txs,
                     const double *tys, const uint64_t *tkeys, const int *tperm, int64_t m,
                     int check, int nout, double *out, int64_t ld_out, cudaStream_t s) {
  if (m == 0) return;
  const TreeDev &td = *b.td;
  PassArgs a{};
  a.th = b.th;
  a.td = b.td;
  EvalItems it;
  eval_items(a, tkeys, m, it, s);
  const BBScale sc = bb_scale(*b.th);
  PhaseTimer timer(PH_EVAL, s);
  const ItemArgs ia{it.items.get(), it.n_items.get(), it.n_items.get() + 1, td.coll.get(),
                    td.bot.get(),   td.top.get(),     txs,                 tys, tperm};
  auto launch = [&](auto pt, auto blocks) {
    using Pol = typename decltype(pt)::type;
    Pol pol{};
    pol.kp = b.kp;
    pol.sx = td.sx.get();
    pol.sy = td.sy.get();
    pol.tau = tau_s;
    pol.check = check;
    pol.out = out;
    pol.ld_out = ld_out;
    pol.p = b.p;
    pol.np = b.np;
    pol.sc = sc;
    pol.xmid = td.xmid.get();
    pol.ymid = td.ymid.get();
    pol.loc = loc;
    constexpr int B = decltype(blocks)::value;
    k_items<Pol, B><<<work_grid(b.th->n_total() + m / EVAL_CHUNK + 1, B), EV_THREADS, 0, s>>>(pol, ia);
  };
  // resident blocks: the Chebyshev values of a target are held in registers
  using P1 = std::integral_constant<int, 6>;
  using P3 = std::integral_constant<int, 4>;
  switch (b.kernel_id) {
    case KERNEL_LAPLACE:
      if (nout == 3)
        launch(TypeOf<BBPolicy<LaplaceF64T, 3>>{}, P3{});
      else
        launch(TypeOf<BBPolicy<LaplaceF64T, 1>>{}, P1{});
      break;
    case KERNEL_MOD_HELMHOLTZ:
      if (nout == 3)
        launch(TypeOf<BBPolicy<ModHelmholtzF64T, 3>>{}, P3{});
      else
        launch(TypeOf<BBPolicy<ModHelmholtzF64T, 1>>{}, P1{});
      break;
    case KERNEL_RADIAL_TABLE:
      FMMB_CHECK(nout == 1, ERR_UNSUPPORTED, "tabulated kernels evaluate potentials only");
      launch(TypeOf<BBPolicy<RadialTableF64, 1>>{}, P1{});
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
  FMMB_CUDA(cudaGetLastError());
}

}  // namespace fmmb
