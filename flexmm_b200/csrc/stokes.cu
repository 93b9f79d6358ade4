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
//  * downward: M2L . source multipoles of all levels (the KIFMM's M2L kernel
//    where a row fits it, np <= 72), then per level += L2LC . parent local
//    (real sibling groups) and the C2E solve, extra unknown dropped
//    (stokes_fmm.py:712-733);
//  * evaluation: (u, v, p) from the leaf's local forces on the large circle
//    (local_expansion_evaluation, stokes_fmm.py:331-360) plus the colleagues'
//    sources (neighbor_evaluation, stokes_fmm.py:361-396).
// A level is one launch each way: its translation and its solve, on the FP64
// tensor cores, on tiles of 8 or 16 rows (k_st_up, k_st_down).  As row GEMMs
// (three launches a level and direction, M2L level by level with 72 columns in
// two tiles of 64) a batch of 12 problems, forward and adjoint, took 1,058
// launches and 6.5 ms; 602 and 3.7 ms now.

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

// log2(r2) and 1 / r2 of a pair
__device__ __forceinline__ void stokes_radial(const LaplaceF64T &K, double r2, double &l2,
                                              double &i2) {
  if (log2_rare_key(r2) < RCP_RARE) {
    l2 = K.at(r2);
    i2 = rcp_newton(r2);
  } else {
    l2 = log2(r2);
    i2 = 1.0 / r2;
  }
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
            stokes_radial(K, fma(dy, dy, dx * dx), l2, i2);
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

  __device__ __forceinline__ bool failed() const { return false; }
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
          stokes_radial(K, r2[r], l2, i2);
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

// ---- level passes: a tile of 8 RB rows, warp w computing column block w ----
constexpr int ST_AHEAD = 8;  // fragment pairs in flight per warp
// threads of the widest row's block (Nequiv 64: 136 columns).  17 warps are five on
// one of the SM's four parts, which holds that many of 96 registers a thread; the
// level kernels take 64 at most by themselves.
constexpr int ST_MAX_THREADS = 544;

// acc[r] += A[8 r ..][.] . B over npairs k pairs of B's column block cb (of nb
// in a k pair); A in shared memory, operator fragments from L2
template <int RB>
__device__ __forceinline__ void st_gemm(const double *A, int lda, const double2 *__restrict__ B,
                                        int nb, int cb, int npairs, double (&acc)[RB][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const double2 *Bp = B + (size_t)cb * 32 + lane;
  const double *Ap = A + g * lda + q;
  double2 f[ST_AHEAD];
#pragma unroll
  for (int i = 0; i < ST_AHEAD; ++i)
    if (i < npairs) f[i] = load_pair(Bp + (size_t)i * nb * 32);
#pragma unroll
  for (int r = 0; r < RB; ++r) acc[r][0] = acc[r][1] = 0.0;
  for (int k0 = 0; k0 < npairs; k0 += ST_AHEAD) {
#pragma unroll
    for (int i = 0; i < ST_AHEAD; ++i) {
      const int kp = k0 + i;
      if (kp < npairs) {
        const double2 b = f[i];
        if (kp + ST_AHEAD < npairs) f[i] = load_pair(Bp + (size_t)(kp + ST_AHEAD) * nb * 32);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          const double *a = Ap + 8 * r * lda + 8 * kp;
          dmma(acc[r], a[0], b.x);
          dmma(acc[r], a[4], b.y);
        }
      }
    }
  }
}

// acc to (ADD: onto) shared rows out[8 RB][ldo], this warp's column block
template <int RB, bool ADD>
__device__ __forceinline__ void st_put(double *out, int ldo, int cb, const double (&acc)[RB][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    double2 *o = reinterpret_cast<double2 *>(out + (8 * r + g) * ldo + 8 * cb + 2 * q);
    double2 v = make_double2(acc[r][0], acc[r][1]);
    if (ADD) {
      const double2 w = *o;
      v = make_double2(w.x + v.x, w.y + v.y);
    }
    *o = v;
  }
}

// x = (P . U) . VHs of the tile's rows, row t to out_row[t] where that is not
// null; T: scratch rows.  The caller synchronises before.
template <int RB>
__device__ __forceinline__ void st_solve(const double2 *U, const double2 *VHs, int np, const double *P,
                                         double *T, double *const *out_row) {
  const int ldp = pad_ld(np), ncb = np / 8, cb = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double acc[RB][2];
  st_gemm<RB>(P, ldp, U, ncb, cb, ncb, acc);
  st_put<RB, false>(T, ldp, cb, acc);
  __syncthreads();
  st_gemm<RB>(T, ldp, VHs, ncb, cb, ncb, acc);
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    double *o = out_row[8 * r + g];
    if (o) *reinterpret_cast<double2 *>(o + 8 * cb + 2 * q) = make_double2(acc[r][0], acc[r][1]);
  }
}

struct StokesLevels {
  const double2 *u[FMM_MAX_LEVELS_DEV], *vhs[FMM_MAX_LEVELS_DEV];
};

// E2C solve of the S2M nodes of all levels: partial check rows -> multipoles
template <int RB>
__global__ void __launch_bounds__(ST_MAX_THREADS)
    k_st_leaves(StokesLevels ops, int np, int L, const int *__restrict__ off,
                            const int *__restrict__ uplist, const int *__restrict__ n_up_ptr,
                            const double *__restrict__ partial, double *__restrict__ mult) {
  constexpr int ROWS = 8 * RB;
  extern __shared__ __align__(16) double smem[];
  __shared__ int node[ROWS], lev[ROWS];
  __shared__ double *orow[ROWS];
  const int ldp = pad_ld(np), n_up = *n_up_ptr, tid = threadIdx.x;
  double *P = smem, *T = P + ROWS * ldp;
  for (int i0 = ROWS * blockIdx.x; i0 < n_up; i0 += ROWS * gridDim.x) {
    const int nloc = min(ROWS, n_up - i0);
    __syncthreads();
    if (tid < ROWS) {
      const int g = tid < nloc ? uplist[i0 + tid] : -1;
      node[tid] = g;
      lev[tid] = g >= 0 ? node_level_of(off, L, g) : -1;
    }
    __syncthreads();
    for (int i = tid; i < ROWS * (np / 2); i += blockDim.x) {
      const int r = i / (np / 2), k = 2 * (i - r * (np / 2));
      if (node[r] >= 0)
        cp_async16(P + r * ldp + k, partial + (size_t)node[r] * np + k);
      else
        P[r * ldp + k] = P[r * ldp + k + 1] = 0.0;
    }
    cp_async_wait_all();
    for (int m = lev[0]; m <= lev[nloc - 1]; ++m) {  // the list is level by level
      __syncthreads();
      if (tid < ROWS) orow[tid] = lev[tid] == m ? mult + (size_t)node[tid] * np : nullptr;
      __syncthreads();
      st_solve<RB>(ops.u[m], ops.vhs[m], np, P, T, orow);
    }
  }
}

// M2M and E2C solve of the parent boxes of one level; their children are the
// contiguous node rows c_first + 4e .. c_first + 4e + 3
template <int RB>
__global__ void k_st_up(StokesArgs::Level op, int np, int c_first, int n_groups,
                        const int *__restrict__ parent, double *mult) {
  constexpr int ROWS = 8 * RB;
  extern __shared__ __align__(16) double smem[];
  __shared__ double *orow[ROWS];
  const int ldp = pad_ld(np), lda = pad_ld(4 * np), ncb = np / 8, tid = threadIdx.x;
  double *P = smem, *T = P + ROWS * ldp, *A = T + ROWS * ldp;
  const int e0 = ROWS * blockIdx.x, nloc = min(ROWS, n_groups - e0);
  if (tid < ROWS)
    orow[tid] = tid < nloc ? mult + (size_t)parent[c_first + 4 * (e0 + tid)] * np : nullptr;
  for (int i = tid + nloc * lda; i < ROWS * lda; i += blockDim.x) A[i] = 0.0;
  pdl_wait();  // the children's multipoles come from the kernels before
  pdl_trigger();
  stage_rows(A, lda, mult + (size_t)(c_first + 4 * e0) * np, nloc, 4 * np);
  cp_async_wait_all();
  __syncthreads();
  double acc[RB][2];
  st_gemm<RB>(A, lda, op.m2m, ncb, tid >> 5, 4 * ncb, acc);
  st_put<RB, false>(P, ldp, tid >> 5, acc);
  __syncthreads();
  st_solve<RB>(op.e2c_u, op.e2c_vhs, np, P, T, orow);
}

// Class c of 8 RB real sibling groups of one level: L2L from their parents
// (l2l not null; stokes_fmm.py:726-733) onto the M2L partial locals, C2E solve
template <int RB>
__global__ void k_st_down(const double2 *c2e_u, const double2 *c2e_vhs, const double2 *l2l, int np,
                          int rg_lo, int rg_cnt, const int *__restrict__ rg,
                          const int *__restrict__ parent, const double *__restrict__ ple,
                          double *loc) {
  constexpr int ROWS = 8 * RB;
  extern __shared__ __align__(16) double smem[];
  __shared__ int node[ROWS], par[ROWS];
  __shared__ double *orow[ROWS];
  const int ldp = pad_ld(np), ncb = np / 8, tid = threadIdx.x, cb = tid >> 5;
  double *P = smem, *T = P + ROWS * ldp, *Lp = T + ROWS * ldp;
  const int q0 = ROWS * (blockIdx.x >> 2), c = blockIdx.x & 3, ngrp = min(ROWS, rg_cnt - q0);
  if (tid < ROWS) {
    const int n = tid < ngrp ? rg[rg_lo + q0 + tid] + c : -1;
    node[tid] = n;
    par[tid] = n >= 0 ? parent[n] : -1;
    orow[tid] = n >= 0 ? loc + (size_t)n * np : nullptr;
  }
  __syncthreads();
  pdl_wait();  // partial locals (M2L) and the parents' locals come from the kernels before
  pdl_trigger();
  for (int i = tid; i < ROWS * (np / 2); i += blockDim.x) {
    const int r = i / (np / 2), k = 2 * (i - r * (np / 2));
    if (node[r] >= 0) {
      cp_async16(P + r * ldp + k, ple + (size_t)node[r] * np + k);
      if (l2l) cp_async16(Lp + r * ldp + k, loc + (size_t)par[r] * np + k);
    } else {
      P[r * ldp + k] = P[r * ldp + k + 1] = 0.0;
      Lp[r * ldp + k] = Lp[r * ldp + k + 1] = 0.0;
    }
  }
  cp_async_wait_all();
  __syncthreads();
  if (l2l) {
    double acc[RB][2];
    st_gemm<RB>(Lp, ldp, l2l, 4 * ncb, c * ncb + cb, ncb, acc);
    st_put<RB, true>(P, ldp, cb, acc);
    __syncthreads();
  }
  st_solve<RB>(c2e_u, c2e_vhs, np, P, T, orow);
}

// two row blocks where one each would fill the SMs more than twice over
int st_rows(int units) { return units > 2 * 148 ? 2 : 1; }

}  // namespace

void run_stokes_upward(const StokesArgs &a, const double *fx, const double *fy, double *partial,
                       double *mult, cudaStream_t s) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  if (th.L < 3) return;
  FMMB_CHECK(th.L <= FMM_MAX_LEVELS_DEV, ERR_INVALID_ARGUMENT, "too many levels");
  const int np = a.np, nthr = 4 * np;  // a warp per column block
  PhaseTimer timer(PH_UPWARD, s);
  auto s2m = a.sgx ? k_stokes_s2m<true> : k_stokes_s2m<false>;
  s2m<<<work_grid(th.n_total(), 8), 128, 0, s>>>(a.neq, np, th.L, circles(a), td.dev_off.get(),
                                                 td.uplist.get(), td.n_up.get(), td.bot.get(),
                                                 td.top.get(), td.xmid.get(), td.ymid.get(),
                                                 td.sx.get(), td.sy.get(), fx, fy, partial, a.sgx,
                                                 a.sgy, a.dnx, a.dny);
  FMMB_CUDA(cudaGetLastError());
  StokesLevels ops{};
  for (int m = 0; m < th.L; ++m) {
    ops.u[m] = a.lev[m].e2c_u;
    ops.vhs[m] = a.lev[m].e2c_vhs;
  }
  const size_t leaf_bytes = sizeof(double) * 32 * pad_ld(np);
  smem_limit(k_st_leaves<2>, leaf_bytes);
  k_st_leaves<2><<<work_grid((th.n_total() + 15) / 16, 4), nthr, leaf_bytes, s>>>(
      ops, np, th.L, td.dev_off.get(), td.uplist.get(), td.n_up.get(), partial, mult);
  FMMB_CUDA(cudaGetLastError());
  for (int m = th.L - 2; m >= 2; --m) {
    const int c_first = th.off[m + 1], n_groups = (th.off[m + 2] - th.off[m + 1]) / 4;
    if (n_groups == 0) continue;
    const int rb = st_rows((n_groups + 7) / 8);
    const size_t bytes = sizeof(double) * 8 * rb * (2 * pad_ld(np) + pad_ld(4 * np));
    auto kern = rb == 1 ? k_st_up<1> : k_st_up<2>;
    smem_limit(kern, bytes);
    launch_pdl(kern, dim3((n_groups + 8 * rb - 1) / (8 * rb)), dim3(nthr), bytes, s, a.lev[m], np,
               c_first, n_groups, td.parent.get(), mult);
  }
}

void run_stokes_downward(const StokesArgs &a, const double *mult, double *ple, double *loc,
                         cudaStream_t s) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  if (th.L < 3) return;
  const int np = a.np, nthr = 4 * np;
  if (np <= ST_M2L_NP) {
    PassArgs pa{};
    pa.np = np;
    pa.td = a.td;
    pa.th = a.th;
    pa.ops_dev = a.ops_dev;
    run_m2l(pa, mult, ple, s);
  } else {  // tiles of one parity class, absent offsets skipped
    PhaseTimer timer(PH_M2L, s);
    for (int m = 2; m < th.L; ++m) {
      const int lo = th.rg_lo[m], n_groups = th.rg_hi[m] - th.rg_lo[m];
      if (n_groups <= 0) continue;
      const int tpc = row_tiles(n_groups);
      rowgemm(M2LRows{td.rg.get(), td.il.get(), mult, lo, n_groups, np, tpc},
              AddGroupRows{td.rg.get(), ple, lo, np}, 4 * tpc, a.lev[m].m2l_cat, np, np, np, s);
    }
  }
  for (int m = 2; m < th.L; ++m) {
    const int lo = th.rg_lo[m], n_groups = th.rg_hi[m] - th.rg_lo[m];
    if (n_groups <= 0) continue;
    PhaseTimer timer(PH_DOWNWARD, s);
    const int rb = st_rows(4 * ((n_groups + 7) / 8));
    const size_t bytes = sizeof(double) * 8 * rb * 3 * pad_ld(np);
    auto kern = rb == 1 ? k_st_down<1> : k_st_down<2>;
    smem_limit(kern, bytes);
    launch_pdl(kern, dim3(4 * ((n_groups + 8 * rb - 1) / (8 * rb))), dim3(nthr), bytes, s,
               a.lev[m].c2e_u, a.lev[m].c2e_vhs, m >= 3 ? a.lev[m - 1].l2l : nullptr, np, lo,
               n_groups, td.rg.get(), td.parent.get(), ple, loc);
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
