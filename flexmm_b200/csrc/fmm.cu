// FMM passes (FP64): upward (S2M / M2M + check-to-equivalent), offset-grouped
// M2L, downward (L2L + check-to-equivalent) and evaluation (L2T + P2P).
//
// Reference path: flexmm/flexmm2d/fmm.py:67-176 (passes), kifmm.py:83-144
// (S2M, C2E, L2T), helpers.py:5-33 (M2L factors), helpers.py:152-194 (P2P).
// Differences of form, not of result:
//  * check-to-equivalent is applied as VH^T diag(1/S) U^T, the factored SVD
//    solve (flexmm/kifmm2d/scalar/helpers.py:240-248), never an explicit
//    inverse; it agrees with the reference's LU solve to ~1e-15;
//  * M2L is target-centric: a tile of 16 to 64 target boxes of one parity class
//    (position inside the parent: 27 of the 40 offsets can occur) gathers the
//    source multipoles that exist at one offset and multiplies them by that
//    offset's operator, accumulating all offsets in shared memory (the
//    reference multiplies every multipole by every offset, then gathers);
//  * the level passes run as one cooperative launch each, tiles of 8 or 16
//    rows of a level against operators held in shared memory;
//  * fake leaves (source-only boxes) get no local expansions: they are never
//    evaluated and never pass anything down;
//  * the GEMMs run on the FP64 tensor cores (mma.sync m8n8k4 f64); the
//    activations sit in shared memory with padded rows (stride 4 mod 16
//    doubles: conflict-free fragment loads), the operators are stored in the
//    order of the fragments their readers need.

#include <algorithm>
#include <type_traits>

#include "fmm.cuh"
#include "gemm.cuh"
#include "radix.cuh"
#include "sweep.cuh"
#include "tcgen05.cuh"
#include "timing.cuh"

namespace fmmb {
namespace {

constexpr int NT = 256;     // threads per tile CTA
constexpr int TCH = EVAL_CHUNK;  // targets per evaluation work item

// the 27 offsets a target can see, by its parity class 2*(ix&1) + (iy&1)
// (offset ids walk ox = -3..3 outer, oy = -3..3 inner, skipping (-1..1)^2)
__constant__ int8_t c_class_off[4][27] = {
    {8, 9, 10, 11, 12, 13, 15, 16, 17, 19, 20, 21, 23, 24, 25, 27, 28, 29, 30, 31, 32, 34, 35, 36, 37, 38, 39},
    {7, 8, 9, 10, 11, 12, 14, 15, 16, 18, 19, 20, 22, 23, 24, 26, 27, 28, 29, 30, 31, 33, 34, 35, 36, 37, 38},
    {1, 2, 3, 4, 5, 6, 8, 9, 10, 11, 12, 13, 15, 16, 17, 19, 20, 21, 23, 24, 25, 27, 28, 29, 30, 31, 32},
    {0, 1, 2, 3, 4, 5, 7, 8, 9, 10, 11, 12, 14, 15, 16, 18, 19, 20, 22, 23, 24, 26, 27, 28, 29, 30, 31}};

// the inverse: class position of offset o in class cls, or -1
__constant__ int8_t c_oi_of[4][40] = {
    {-1, -1, -1, -1, -1, -1, -1, -1, 0, 1, 2, 3, 4, 5, -1, 6, 7, 8, -1, 9, 10, 11, -1, 12, 13, 14, -1, 15, 16, 17, 18, 19, 20, -1, 21, 22, 23, 24, 25, 26},
    {-1, -1, -1, -1, -1, -1, -1, 0, 1, 2, 3, 4, 5, -1, 6, 7, 8, -1, 9, 10, 11, -1, 12, 13, 14, -1, 15, 16, 17, 18, 19, 20, -1, 21, 22, 23, 24, 25, 26, -1},
    {-1, 0, 1, 2, 3, 4, 5, -1, 6, 7, 8, 9, 10, 11, -1, 12, 13, 14, -1, 15, 16, 17, -1, 18, 19, 20, -1, 21, 22, 23, 24, 25, 26, -1, -1, -1, -1, -1, -1, -1},
    {0, 1, 2, 3, 4, 5, -1, 6, 7, 8, 9, 10, 11, -1, 12, 13, 14, -1, 15, 16, 17, -1, 18, 19, 20, -1, 21, 22, 23, 24, 25, 26, -1, -1, -1, -1, -1, -1, -1, -1}};

// the factor a kernel's loops fold into their staged charges and locals
template <class KF, bool kFolded>
__device__ __forceinline__ double fold_of() {
  if constexpr (kFolded)
    return KF::kFold;
  else
    return 1.0;
}

// ---------------------------------------------------------------- upward ----
__device__ __forceinline__ int level_of_node(const int *__restrict__ off, int L, int g) {
  int lo = 0, hi = L;  // largest l with off[l] <= g
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= g)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// first of n consecutive places taken from *next for every lane of the warp
// (one atomic for all; all lanes must call)
__device__ __forceinline__ int warp_place(int n, int *next) {
  const int lane = threadIdx.x & 31;
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  int base = 0;
  if (lane == 31 && incl > 0) base = atomicAdd(next, incl);
  return __shfl_sync(0xffffffffu, base, 31) + incl - n;
}

// S2M of every S2M node (leaves holding points, levels >= 2) of every level in
// one launch (flexmm/flexmm2d/kifmm.py:96-105): a warp sums one node's sources
// into its check potentials, written into the node's multipole row; the
// check-to-equivalent solve follows in place (k_c2e_leaves), apart from it so
// that a block needs no room for operators here and many warps hide the loads.
// The lanes are check points, two each where there are more than 48, one each
// for the first 32 and G lanes each for up to 16 more; the sweep is the
// evaluation's (sweep.cuh).  Bound by the FP64 pipe, with the log table's reads.
// 1M clustered points, Nequiv 60: 120 us and 58 for the solve, where one kernel
// of 32-node tiles took 250; 250k points on rings, Nequiv 40: 28 + 14 after 64.
constexpr int S2M_WARPS = 4, S2M_CHUNK = 64;  // sources staged per warp

template <class KF, bool DIP>
__global__ void __launch_bounds__(32 * S2M_WARPS, 8)
    k_s2m(KernelParams kp, int neq, int np, int L, const int *__restrict__ off,
          const int *__restrict__ uplist, const int *__restrict__ n_up_ptr,
          const int *__restrict__ bot, const int *__restrict__ top,
          const double *__restrict__ xmid, const double *__restrict__ ymid,
          const double *__restrict__ sx, const double *__restrict__ sy,
          const double *__restrict__ tau, const LevelOpsDev *__restrict__ ops,
          double *__restrict__ mult, const double *__restrict__ dvx,
          const double *__restrict__ dvy) {
  __shared__ double2 s_xy[S2M_WARPS][S2M_CHUNK], s_dv[DIP ? S2M_WARPS : 1][S2M_CHUNK];
  __shared__ double s_q[S2M_WARPS][S2M_CHUNK];
  __shared__ FunctorSmem<KF> fsm;
  KF K(kp);
  fsm.bind(K);
  const double fold = fold_of<KF, KF::kLogTable>();
  const int n_up = *n_up_ptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = blockIdx.x * S2M_WARPS + warp; i < n_up; i += gridDim.x * S2M_WARPS) {
    const int node = uplist[i];
    const LevelOpsDev &op = ops[level_of_node(off, L, node)];
    const int b = bot[node], e = top[node];
    const double cx = xmid[node], cy = ymid[node];
    double *row = mult + (size_t)node * np;
    int staged = -1;
    auto points = [&](auto rc, int k0, int G) {  // R tiles of check points from k0 on
      constexpr int R = decltype(rc)::value;
      const int sub = lane & (G - 1), k = k0 + lane / G;
      double x[R], y[R], v[R][2];
      long long none[R] = {};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        x[r] = op.lx[min(k + 32 * r, neq - 1)];
        y[r] = op.ly[min(k + 32 * r, neq - 1)];
        v[r][0] = v[r][1] = 0.0;
      }
      for (int j0 = b; j0 < e; j0 += S2M_CHUNK) {
        const int nj = min(S2M_CHUNK, e - j0);
        if (staged != j0) {
          __syncwarp();
          for (int j = lane; j < nj; j += 32) {
            s_xy[warp][j] = make_double2(sx[j0 + j] - cx, sy[j0 + j] - cy);
            s_q[warp][j] = tau[j0 + j] * fold;
            if constexpr (DIP) s_dv[warp][j] = make_double2(dvx[j0 + j], dvy[j0 + j]);
          }
          __syncwarp();
          staged = j0;
        }
        pot_sweep<KF, R, DIP, false>(K, s_xy[warp], s_q[warp], s_dv[DIP ? warp : 0], nullptr, x, y,
                                     none, sub, nj, G, 0, v);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double o = v[r][0] + v[r][1];
        if (R == 1)
          for (int w = G >> 1; w >= 1; w >>= 1) o += __shfl_xor_sync(0xffffffffu, o, w);
        if (sub == 0 && k + 32 * r < neq) row[k + 32 * r] = o;
      }
    };
    if (neq + lane < np) row[neq + lane] = 0.0;  // (np - neq < 8)
    using One = std::integral_constant<int, 1>;
    if (neq > 48) {
      points(std::integral_constant<int, 2>{}, 0, 1);
    } else {
      int k = 0;
      if (neq >= 32) {
        points(One{}, 0, 1);
        k = 32;
      }
      if (k < neq) {
        int G = 1;
        while (2 * G * (neq - k) <= 32) G *= 2;
        points(One{}, k, G);
      }
    }
  }
}

// The same for up to S2M_COLS charge columns at a time (column group
// blockIdx.y): each kernel value is computed once for all of them.  16 columns
// at 60k points on a ring, K0: 72 us, and 510 us a column at a time.
constexpr int S2M_COLS = 8;
template <class KF>
__global__ void __launch_bounds__(32 * S2M_WARPS, 6)
    k_s2m_multi(KernelParams kp, int neq, int np, int L, const int *__restrict__ off,
                const int *__restrict__ uplist, const int *__restrict__ n_up_ptr,
                const int *__restrict__ bot, const int *__restrict__ top,
                const double *__restrict__ xmid, const double *__restrict__ ymid,
                const double *__restrict__ sx, const double *__restrict__ sy,
                const double *__restrict__ tau, const LevelOpsDev *__restrict__ ops,
                double *__restrict__ mult, int n_rhs, int64_t tstride, int64_t cstride) {
  __shared__ double2 s_xy[S2M_WARPS][32];
  __shared__ double s_q[S2M_WARPS][32][S2M_COLS];
  __shared__ FunctorSmem<KF> fsm;
  KF K(kp);
  fsm.bind(K);
  const double fold = fold_of<KF, KF::kLogTable>();
  const int c0 = S2M_COLS * blockIdx.y, ncol = min(S2M_COLS, n_rhs - c0);
  tau += c0 * tstride;
  mult += c0 * cstride;
  const int n_up = *n_up_ptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = blockIdx.x * S2M_WARPS + warp; i < n_up; i += gridDim.x * S2M_WARPS) {
    const int node = uplist[i];
    const LevelOpsDev &op = ops[level_of_node(off, L, node)];
    const int b = bot[node], e = top[node];
    const double cx = xmid[node], cy = ymid[node];
    if (neq + lane < np)
      for (int c = 0; c < ncol; ++c) mult[c * cstride + (size_t)node * np + neq + lane] = 0.0;
    for (int k0 = 0; k0 < neq; k0 += 32) {
      int G = 1;
      while (2 * G * (neq - k0) <= 32) G *= 2;
      const int sub = lane & (G - 1), k = k0 + lane / G;
      const double x = op.lx[min(k, neq - 1)], y = op.ly[min(k, neq - 1)];
      double v[S2M_COLS] = {};
      for (int j0 = b; j0 < e; j0 += 32) {
        const int nj = min(32, e - j0);
        __syncwarp();
        if (lane < nj) {
          s_xy[warp][lane] = make_double2(sx[j0 + lane] - cx, sy[j0 + lane] - cy);
#pragma unroll
          for (int c = 0; c < S2M_COLS; ++c)
            s_q[warp][lane][c] = c < ncol ? tau[c * tstride + j0 + lane] * fold : 0.0;
        }
        __syncwarp();
#pragma unroll 2
        for (int j = sub; j < nj; j += G) {
          const double dx = x - s_xy[warp][j].x, dy = y - s_xy[warp][j].y;
          double kv;
          if constexpr (KF::kLogTable)
            kv = K.raw(dx, dy);
          else
            kv = K(0.0, 0.0, dx, dy);
#pragma unroll
          for (int c = 0; c < S2M_COLS; ++c) v[c] = fma(kv, s_q[warp][j][c], v[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < S2M_COLS; ++c) {
        double o = v[c];
        for (int w = G >> 1; w >= 1; w >>= 1) o += __shfl_xor_sync(0xffffffffu, o, w);
        if (sub == 0 && k < neq && c < ncol) mult[c * cstride + (size_t)node * np + k] = o;
      }
    }
  }
}

// The level passes run as one cooperative launch each (upward, downward), one
// block per SM, the levels in turn with a grid barrier between them.  A level
// is a short chain (its inputs from L2, three GEMMs on the FP64 tensor cores,
// its outputs), bound by latency: as a launch of its own it took 26 us at 250k
// ring points, Nequiv 40 (operators copied through shared memory 16 rows at a
// time), and with the operators read from L2 as fragments 11 us (one SM reads
// 13 bytes a clock with four loads in flight per warp, and a new
// launch fetches its instructions again).  So a block keeps a
// level's operators in shared memory, copied while it is still busy with the
// level before (the translation's as soon as its last tile is through it, U
// and VH at the level's end); between levels it waits for the grid barrier
// (2,500 clocks) and its first inputs only.  Both passes: 470 -> 195 us at 250k
// ring points (19 levels), 838 -> 304 us at 1M clustered points, Nequiv 60.
struct LevelSpan {
  int first, count;  // first child node (upward) or real group (downward); groups
  int rb, tiles;     // row blocks (of 8 groups) per tile; tiles per charge column
};
struct LevelSpans {
  int m0, n;  // levels m0, m0 + step, ... (n of them)
  LevelSpan lv[FMM_MAX_LEVELS_DEV];
};

// Row blocks per tile of a level of `units` 8-group row blocks on `grid`
// blocks.  A tile takes about as long with two row blocks as with one (its
// chain of DMMAs waits on itself): two where that saves a round.
int level_rows(int64_t units, int64_t grid, int rb_max) {
  const int64_t one = (units + grid - 1) / grid, two = (units + 2 * grid - 1) / (2 * grid);
  return rb_max >= 2 && 1.15 * double(two) < double(one) ? 2 : 1;
}

// A level's operators in shared memory, filled by bulk copies (one thread
// starts them: copied by all threads in 16-byte pieces they held the block up
// for 3,400 clocks a level at Nequiv 40) that two mbarriers count: M by
// bar[0], U, VH and 1/S by bar[1].
struct LevelStage {
  double2 *M, *U, *V;  // translation (M2M, or L2L of one class), U, VH fragments
  double *sinv;        // [np] 1/S
  int np;
  uint64_t *bar;
  // called by one thread, after a block barrier behind the last read
  __device__ void load_uv(const LevelOpsDev &op) const {
    const uint32_t sq = 8u * np * np;
    bulk_expect(bar + 1, 2 * sq + 8u * np);
    bulk_copy(U, op.u_f, sq, bar + 1);
    bulk_copy(V, op.vh_f, sq, bar + 1);
    bulk_copy(sinv, op.sinv, 8u * np, bar + 1);
  }
  // wait for the k-th filling of both; false when the wait ran out
  __device__ bool wait(uint32_t k) const {
    return tc::mbar_wait(tc::smem_u32(bar), k & 1u, LEVEL_WAIT_TRIES) &&
           tc::mbar_wait(tc::smem_u32(bar + 1), k & 1u, LEVEL_WAIT_TRIES);
  }
  static constexpr uint32_t LEVEL_WAIT_TRIES = 1u << 20;
};
// doubles of a stage whose translation has m_blocks np x np blocks
__host__ __device__ inline size_t level_ops_doubles(int np, int m_blocks) {
  return (size_t)(2 + m_blocks) * np * np + 64;
}
__device__ inline LevelStage level_stage(double *smem, int np, int m_blocks, uint64_t *bar) {
  double2 *p = reinterpret_cast<double2 *>(smem);
  LevelStage st;
  st.np = np;
  st.M = p;
  st.U = p + m_blocks * np * np / 2;
  st.V = st.U + np * np / 2;
  st.sinv = reinterpret_cast<double *>(st.V + np * np / 2);
  st.bar = bar;
  if (threadIdx.x == 0) {
    tc::mbar_init(tc::smem_u32(bar), 1);
    tc::mbar_init(tc::smem_u32(bar + 1), 1);
    tc::fence_mbar_init();
  }
  __syncthreads();
  return st;
}

constexpr int LEVEL_RB = 2;  // most row blocks per tile (4: 649 us for 609 at 100k uniform points)
struct LevelSmem {           // static shared memory of a level kernel
  double part[FG_PART];
  double *orow[2][8 * LEVEL_RB];
  uint64_t bar[2];
};

size_t up_smem(int np, int rb) {
  return sizeof(double) *
         (level_ops_doubles(np, 4) + (size_t)8 * rb * (2 * (size_t)pad_ld(np) + pad_ld(4 * np)));
}

// M2M + C2E of one level (flexmm/flexmm2d/fmm.py:91-98): a tile is 8 RB parent
// groups, whose children are the contiguous node rows first + 4e ..
// first + 4e + 3 of the level below.  P[t] = M2MC . children.  The next tile's
// children are copied while the tile is in its check-to-equivalent solve;
// next_ops() starts the copies of the operators of the block's next level.
template <int RB, class F>
__device__ __forceinline__ void up_level(const LevelStage &st, const LevelSpan &lv, int n_rhs,
                                         const int *__restrict__ parent, double *mult,
                                         int64_t cstride, double *rows, LevelSmem &sm, F &&next_ops) {
  constexpr int ROWS = 8 * RB;
  const int np = st.np, ldp = pad_ld(np), lda = pad_ld(4 * np), ncb = np / 8;
  double *P = rows;           // [ROWS][ldp] check potentials
  double *T = P + ROWS * ldp;  // [ROWS][ldp] C2E scratch
  double *A = T + ROWS * ldp;  // [ROWS][lda] children multipoles
  const UnitSplit<RB> t(ncb);
  const int64_t total = (int64_t)lv.tiles * n_rhs;
  auto load_a = [&](int64_t u, int slot) {  // the tile's inputs (one copy group) and outputs
    const int col = int(u / lv.tiles), e0 = ROWS * int(u - (int64_t)col * lv.tiles);
    const int nloc = min(ROWS, lv.count - e0);
    double *mu = mult + col * cstride;
    if (threadIdx.x < ROWS)
      sm.orow[slot][threadIdx.x] =
          (int)threadIdx.x < nloc
              ? mu + (size_t)parent[lv.first + 4 * (e0 + (int)threadIdx.x)] * np
              : nullptr;
    for (int j = threadIdx.x + nloc * lda; j < ROWS * lda; j += NT) A[j] = 0.0;
    stage_rows(A, lda, mu + (size_t)(lv.first + 4 * e0) * np, nloc, 4 * np);
    cp_async_commit_group();
  };
  int slot = 0;
  load_a(blockIdx.x, 0);
  for (int64_t u = blockIdx.x; u < total; u += gridDim.x, slot ^= 1) {
    cp_async_wait_all();
    __syncthreads();
    double acc[RB][2];
    unit_gemm(t, A, lda, st.M, ncb, 4 * ncb, acc);
    unit_sum(t, acc, sm.part);
    unit_each(t, acc, [&](int r, int c, double a, double b) {
      *reinterpret_cast<double2 *>(P + r * ldp + c) = make_double2(a, b);
    });
    __syncthreads();
    if (u + gridDim.x < total)
      load_a(u + gridDim.x, slot ^ 1);
    else if (threadIdx.x == 0)
      next_ops();
    c2e_rows_smem<RB>(st.U, st.V, st.sinv, np, P, T, sm.part, sm.orow[slot]);
  }
}

// the first level from i on in which this block has a tile
__device__ __forceinline__ int next_level(const LevelSpans &sp, int i, int n_rhs) {
  while (i < sp.n && (int64_t)sp.lv[i].tiles * n_rhs <= blockIdx.x) ++i;
  return i;
}

__global__ void __launch_bounds__(NT, 2) k_up_levels(LevelSpans sp, int np, int n_rhs,
                                                  const int *__restrict__ parent,
                                                  const LevelOpsDev *__restrict__ ops, double *mult,
                                                  int64_t cstride, RadixSync *sync, int *fail) {
  extern __shared__ __align__(16) double smem[];
  __shared__ __align__(16) LevelSmem sm;
  const LevelStage st = level_stage(smem, np, 4, sm.bar);
  double *rows = smem + level_ops_doubles(np, 4);
  int nxt = next_level(sp, 0, n_rhs);  // the level whose operators are (being) staged
  uint32_t fills = 0;
  auto load_m = [&] {
    if (nxt >= sp.n) return;
    bulk_expect(sm.bar, 32u * np * np);
    bulk_copy(st.M, ops[sp.m0 - nxt].m2m_f, 32u * np * np, sm.bar);
  };
  if (threadIdx.x == 0 && nxt < sp.n) {
    load_m();
    st.load_uv(ops[sp.m0 - nxt]);
  }
  for (int i = 0; i < sp.n; ++i) {
    const LevelSpan lv = sp.lv[i];
    if (i == nxt) {
      nxt = next_level(sp, i + 1, n_rhs);
      if (!__syncthreads_and(st.wait(fills++))) {
        if (threadIdx.x == 0) atomicExch(fail, 1);
        return;
      }
      if (lv.rb == 1)
        up_level<1>(st, lv, n_rhs, parent, mult, cstride, rows, sm, load_m);
      else
        up_level<2>(st, lv, n_rhs, parent, mult, cstride, rows, sm, load_m);
      if (nxt < sp.n) {
        __syncthreads();  // U and VH have been read
        if (threadIdx.x == 0) st.load_uv(ops[sp.m0 - nxt]);
      }
    }
    if (i + 1 < sp.n && !grid_barrier(sync, fail)) {
      if (nxt < sp.n) st.wait(fills);  // the copies in flight
      return;
    }
  }
}

// Check-to-equivalent of the S2M nodes' rows (check potentials, from S2M) in
// place, all levels and charge columns in one launch.  A block takes a
// contiguous run of the level-major list, so it stages a level's operators
// once or twice, and reads the next tile of 16 rows during the current one.
// Bound by the DMMA pipe and, at few tiles, by staging the operators.
constexpr int C2E_RB = 2, C2E_ROWS = 8 * C2E_RB;
size_t c2e_leaves_smem(int np) {
  return sizeof(double) * (level_ops_doubles(np, 0) + (size_t)3 * C2E_ROWS * pad_ld(np));
}
__global__ void __launch_bounds__(NT, 2) k_c2e_leaves(int np, int L, int n_rhs,
                                                      const int *__restrict__ off,
                                                      const int *__restrict__ uplist,
                                                      const int *__restrict__ n_up_ptr,
                                                      const LevelOpsDev *__restrict__ ops,
                                                      double *mult, int64_t cstride) {
  extern __shared__ __align__(16) double smem[];
  __shared__ __align__(16) double part[FG_PART];
  __shared__ double *orow[C2E_ROWS];
  __shared__ int node[2][C2E_ROWS], lev[2][C2E_ROWS];
  const int ldp = pad_ld(np), tid = threadIdx.x, n_up = *n_up_ptr;
  double2 *U = reinterpret_cast<double2 *>(smem), *V = U + np * np / 2;
  double *sinv = reinterpret_cast<double *>(V + np * np / 2);
  double *T = smem + level_ops_doubles(np, 0), *P[2] = {T + C2E_ROWS * ldp, T + 2 * C2E_ROWS * ldp};
  const int tiles = (n_up + C2E_ROWS - 1) / C2E_ROWS;
  const int64_t total = (int64_t)tiles * n_rhs;
  const int64_t u0 = total * blockIdx.x / gridDim.x, u1 = total * (blockIdx.x + 1) / gridDim.x;
  auto load = [&](int64_t u, int slot) {  // the tile's nodes, then their rows (a copy group)
    const int col = int(u / tiles), i0 = C2E_ROWS * int(u - (int64_t)col * tiles);
    if (tid < C2E_ROWS) {
      const int g = i0 + tid < n_up ? uplist[i0 + tid] : -1;
      node[slot][tid] = g;
      lev[slot][tid] = g >= 0 ? level_of_node(off, L, g) : -1;
    }
    for (int i = tid; i < C2E_ROWS * (np / 2); i += NT) {
      const int r = i / (np / 2), k = 2 * (i - r * (np / 2));
      if (i0 + r < n_up)
        cp_async16(P[slot] + r * ldp + k, mult + col * cstride + (size_t)uplist[i0 + r] * np + k);
      else
        P[slot][r * ldp + k] = P[slot][r * ldp + k + 1] = 0.0;
    }
    cp_async_commit_group();
  };
  int have = -1, slot = 0;  // level whose operators are staged
  if (u0 < u1) load(u0, 0);
  for (int64_t u = u0; u < u1; ++u, slot ^= 1) {
    const int col = int(u / tiles);
    cp_async_wait_all();
    __syncthreads();
    if (u + 1 < u1) load(u + 1, slot ^ 1);
    const int nloc = min(C2E_ROWS, n_up - C2E_ROWS * int(u - (int64_t)col * tiles));
    for (int m = lev[slot][0]; m <= lev[slot][nloc - 1]; ++m) {
      if (tid < C2E_ROWS)
        orow[tid] = lev[slot][tid] == m ? mult + col * cstride + (size_t)node[slot][tid] * np : nullptr;
      if (m != have) {
        for (int j = tid; j < np * np / 2; j += NT) {
          cp_async16(U + j, ops[m].u_f + j);
          cp_async16(V + j, ops[m].vh_f + j);
        }
        if (tid < np) sinv[tid] = ops[m].sinv[tid];
        cp_async_commit_group();
        cp_async_wait_all();
        have = m;
      }
      __syncthreads();
      c2e_rows_smem<C2E_RB>(U, V, sinv, np, P[slot], T, part, orow);
      __syncthreads();  // operators, T and orow are free
    }
  }
}

// ------------------------------------------------------------------- M2L ----
struct M2LTiles {
  int n_levels;
  int tile_start[4 * FMM_MAX_LEVELS_DEV + 1];  // first tile of each (level, parity class)
  int rg_lo[FMM_MAX_LEVELS_DEV];               // real groups of each level
  int rg_cnt[FMM_MAX_LEVELS_DEV];
};

// One tile = up to tt targets of one parity class of one level (the 27 offsets
// that class can see).  Per offset, the targets that have a source there are
// listed; their source multipoles are gathered next to one another and
// multiplied by the offset's operator 8 rows at a time, and each product row is
// added to its target's row of partial locals in shared memory.  So the
// tensor cores see the interactions that exist, rounded up to 8 per offset and
// tile: on a ring of points a target has a fraction of its 27 sources, and a
// tile that multiplies every target's row for every offset (as this kernel did)
// works on zeros.  250k ring points, Nequiv 40: 370 -> 110 us; 16 columns there
// 2,910 -> 500; 1M clustered, Nequiv 60: 735 -> 437; 100k uniform, Nequiv 32:
// 70 -> 34; 3k, Nequiv 16: 45 -> 24.  The row order of a list does not matter: a row's sum runs over the
// offsets in order.
// Warp w owns column block w (8 columns) of every row, so rows are updated
// without conflicts and one barrier per offset (its gather has arrived, the
// buffer before is free) is all there is.  The operator is read as fragments:
// into registers, one offset ahead; at np <= 16, where an offset is over before
// an L2 read returns, through the gather's ring of buffers, three ahead.
// Factored (SVD) operators are multiplied out on the host: at the ranks the
// reference's rule factors (below Nequiv / 2, rounded up to 8) two thin products
// cost as much as the full one.
template <int NCB>
struct M2LShape {
  static constexpr int np = 8 * NCB, ldp = np + 4;
  static constexpr bool kOpInRing = NCB <= 2;
  static constexpr int kStages = NCB <= 2 ? 4 : NCB <= 4 ? 3 : 2;
  static constexpr int kTargets = NCB <= 4 || NCB > 8 ? 32 : 64;  // targets per tile
  static constexpr int kBlocks = NCB > 6 ? 2 : NCB > 4 ? 3 : NCB > 2 ? 6 : 8;  // resident per SM
  static __host__ __device__ size_t stage_doubles(int tt) {
    return (size_t)tt * ldp + (kOpInRing ? np * np : 0);
  }
  static __host__ __device__ size_t smem(int tt) {
    return 8 * (tt * ldp + kStages * stage_doubles(tt)) + 27 * tt * (sizeof(int) + 1);
  }
};

template <int NCB>
__global__ void __launch_bounds__(32 * NCB, M2LShape<NCB>::kBlocks)
    k_m2l(M2LTiles tiles, int tt, const int *__restrict__ rg, const int *__restrict__ il,
          const LevelOpsDev *__restrict__ ops, const double *__restrict__ mult,
          double *__restrict__ ple, int64_t cstride) {
  using Sh = M2LShape<NCB>;
  constexpr int np = Sh::np, ldp = Sh::ldp, S = Sh::kStages, nthr = 32 * NCB;
  mult += blockIdx.y * cstride;  // charge column blockIdx.y
  ple += blockIdx.y * cstride;
  extern __shared__ __align__(16) double smem[];
  double *acc = smem;                 // [tt][ldp] partial locals
  double *ring = acc + tt * ldp;      // stages: [tt][ldp] gathered multipoles (, operator)
  const size_t stage = Sh::stage_doubles(tt);
  int *l_src = reinterpret_cast<int *>(ring + S * stage);      // [27][tt] source nodes
  uint8_t *l_row = reinterpret_cast<uint8_t *>(l_src + 27 * tt);  // [27][tt] target rows
  __shared__ int l_n[27], s_act[27], s_nact;
  __shared__ const double2 *s_op[27];  // the active offsets' operators
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  // this block's (level, parity class, range of real groups)
  int slot = 0;
  while (slot + 1 < 4 * tiles.n_levels && tiles.tile_start[slot + 1] <= (int)blockIdx.x) ++slot;
  const int m = slot >> 2, cls = slot & 3;
  const int q0 = tt * (blockIdx.x - tiles.tile_start[slot]);
  const int nloc = min(tt, tiles.rg_cnt[m] - q0);
  const int *tgt = rg + tiles.rg_lo[m] + q0;  // target t: node tgt[t] + cls
  const LevelOpsDev &op = ops[m];
  if (tid < 27) l_n[tid] = 0;
  for (int i = tid; i < tt * ldp; i += nthr) acc[i] = 0.0;
  __syncthreads();
  for (int t0 = 32 * warp; t0 < nloc; t0 += nthr) {  // lists: a warp lists 32 targets
    const int t = t0 + lane;
    int row[N_OFFSETS];
    const int4 *ilr =
        reinterpret_cast<const int4 *>(il + (size_t)(t < nloc ? tgt[t] + cls : 0) * N_OFFSETS);
#pragma unroll
    for (int i = 0; i < N_OFFSETS / 4; ++i) {
      const int4 v = t < nloc ? __ldg(ilr + i) : make_int4(-1, -1, -1, -1);
      row[4 * i] = v.x;
      row[4 * i + 1] = v.y;
      row[4 * i + 2] = v.z;
      row[4 * i + 3] = v.w;
    }
#pragma unroll
    for (int o = 0; o < N_OFFSETS; ++o) {
      const int oi = c_oi_of[cls][o];
      if (oi < 0 || op.kind[o] == M2L_NULL) continue;  // the same for all lanes
      const unsigned has = __ballot_sync(0xffffffffu, row[o] >= 0);
      if (!has) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(&l_n[oi], __popc(has));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(has & ((1u << lane) - 1u));
      if (row[o] >= 0) {
        l_src[oi * tt + at] = row[o];
        l_row[oi * tt + at] = (uint8_t)t;
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    const unsigned act = __ballot_sync(0xffffffffu, lane < 27 && l_n[lane < 27 ? lane : 0] > 0);
    if (lane < 27 && (act >> lane & 1u)) {
      const int at = __popc(act & ((1u << lane) - 1u));
      s_act[at] = lane;
      s_op[at] = op.m2l_f[c_class_off[cls][lane]];
    }
    if (lane == 0) s_nact = __popc(act);
  }
  __syncthreads();
  const int nact = s_nact;
  auto gather = [&](int a) {  // active offset a into its ring stage (one copy group)
    if (a < nact) {
      const int oi = s_act[a], n = l_n[oi];
      double *G = ring + (a % S) * stage;
      for (int i = tid; i < n * (np / 2); i += nthr) {
        const int r = i / (np / 2), k = 2 * (i - r * (np / 2));
        cp_async16(G + r * ldp + k, mult + (size_t)l_src[oi * tt + r] * np + k);
      }
      if (Sh::kOpInRing) {
        const double2 *B = s_op[a];
        double2 *D = reinterpret_cast<double2 *>(G + tt * ldp);
        for (int i = tid; i < np * np / 2; i += nthr) cp_async16(D + i, B + i);
      }
    }
    cp_async_commit_group();
  };
  double2 b[NCB], bn[Sh::kOpInRing ? 1 : NCB];  // this warp's operator fragments, and the next ones
  auto load_op = [&](int a, double2 (&v)[Sh::kOpInRing ? 1 : NCB]) {
    if constexpr (!Sh::kOpInRing) {
      const double2 *B = s_op[a] + warp * 32 + lane;
#pragma unroll
      for (int kp = 0; kp < NCB; ++kp) v[kp] = load_pair(B + kp * NCB * 32);
    }
  };
#pragma unroll
  for (int a = 0; a < S - 1; ++a) gather(a);
  if (nact > 0) load_op(0, bn);
  for (int a = 0; a < nact; ++a) {
    cp_async_wait_group<S - 2>();
    __syncthreads();  // offset a is there, and the stage of offset a - 1 has been read
    gather(a + S - 1);
    const int oi = s_act[a], n = l_n[oi];
    const double *G = ring + (a % S) * stage;
    if constexpr (Sh::kOpInRing) {
      const double2 *D = reinterpret_cast<const double2 *>(G + tt * ldp) + warp * 32 + lane;
#pragma unroll
      for (int kp = 0; kp < NCB; ++kp) b[kp] = D[kp * NCB * 32];
    } else {
#pragma unroll
      for (int kp = 0; kp < NCB; ++kp) b[kp] = bn[kp];
      if (a + 1 < nact) load_op(a + 1, bn);
    }
    for (int r0 = 0; r0 < n; r0 += 16) {  // two row blocks: two chains of DMMAs
      const bool two = r0 + 8 < n;
      const int ra = r0 + g, rb = r0 + 8 + g;
      double *oa = acc + l_row[oi * tt + min(ra, n - 1)] * ldp + 8 * warp + 2 * q;
      double *ob = acc + l_row[oi * tt + min(rb, n - 1)] * ldp + 8 * warp + 2 * q;
      const double *A0 = G + ra * ldp + q, *A1 = two ? A0 + 8 * ldp : A0;
      double2 va = *reinterpret_cast<const double2 *>(oa);
      double2 vb = *reinterpret_cast<const double2 *>(ob);
      double c0[2] = {va.x, va.y}, c1[2] = {vb.x, vb.y};
#pragma unroll
      for (int kp = 0; kp < NCB; ++kp) {
        dmma(c0, A0[8 * kp], b[kp].x);
        if (two) dmma(c1, A1[8 * kp], b[kp].x);
        dmma(c0, A0[8 * kp + 4], b[kp].y);
        if (two) dmma(c1, A1[8 * kp + 4], b[kp].y);
      }
      // (rows past the list hold leftovers: a product row depends on its own
      // row only, and these are not stored)
      if (ra < n) *reinterpret_cast<double2 *>(oa) = make_double2(c0[0], c0[1]);
      if (rb < n) *reinterpret_cast<double2 *>(ob) = make_double2(c1[0], c1[1]);
    }
  }
  __syncthreads();
  for (int i = tid; i < nloc * (np / 2); i += nthr) {
    const int t = i / (np / 2), k = 2 * (i - t * (np / 2));
    *reinterpret_cast<double2 *>(ple + (size_t)(tgt[t] + cls) * np + k) =
        *reinterpret_cast<const double2 *>(acc + t * ldp + k);
  }
}

// -------------------------------------------------------------- downward ----
size_t down_smem(int np, int rb) {
  return sizeof(double) * (level_ops_doubles(np, 1) + (size_t)8 * rb * 5 * pad_ld(np));
}

// One level: a tile is class c (child c) of 8 RB real sibling groups: L2L from
// their parents (has_l2l; flexmm/flexmm2d/fmm.py:140-147), plus the M2L partial
// locals, then check-to-equivalent.  Block b takes class b mod 4 in every
// level (the grid is a multiple of 4), so it stages a quarter of the L2L
// operator only.
template <int RB, class F>
__device__ __forceinline__ void down_level(const LevelStage &st, const LevelSpan &lv, int n_rhs,
                                           bool has_l2l, const int *__restrict__ rg,
                                           const int *__restrict__ parent,
                                           const double *__restrict__ ple, double *loc,
                                           int64_t cstride, double *rows, LevelSmem &sm,
                                           F &&next_ops) {
  constexpr int ROWS = 8 * RB;
  const int np = st.np, ldp = pad_ld(np), ncb = np / 8, c = blockIdx.x & 3;
  double *T = rows;                                            // [ROWS][ldp] C2E scratch
  double *PL[2] = {T + ROWS * ldp, T + 3 * ROWS * ldp};  // per slot: partial locals, parents' locals
  const UnitSplit<RB> t(ncb);
  const int64_t total = (int64_t)lv.tiles * n_rhs;  // tiles of this class
  const int64_t step = gridDim.x / 4, u0 = blockIdx.x / 4;
  auto load_rows = [&](int64_t u, int slot) {
    const int col = int(u / lv.tiles), q0 = ROWS * int(u - (int64_t)col * lv.tiles);
    const int ngrp = min(ROWS, lv.count - q0);
    double *lo = loc + col * cstride, *P = PL[slot], *Lp = P + ROWS * ldp;
    const double *pl = ple + col * cstride;
    for (int j = threadIdx.x; j < ROWS * (np / 2); j += NT) {
      const int r = j / (np / 2), k = 2 * (j - r * (np / 2));
      if (r < ngrp) {
        const int n = rg[lv.first + q0 + r] + c;
        cp_async16(P + r * ldp + k, pl + (size_t)n * np + k);
        if (has_l2l) cp_async16(Lp + r * ldp + k, lo + (size_t)parent[n] * np + k);
        if (k == 0) sm.orow[slot][r] = lo + (size_t)n * np;
      } else {
        P[r * ldp + k] = P[r * ldp + k + 1] = 0.0;
        Lp[r * ldp + k] = Lp[r * ldp + k + 1] = 0.0;
        if (k == 0) sm.orow[slot][r] = nullptr;
      }
    }
    cp_async_commit_group();
  };
  int slot = 0;
  load_rows(u0, 0);
  for (int64_t u = u0; u < total; u += step, slot ^= 1) {
    const bool last = u + step >= total;
    double *P = PL[slot], *Lp = P + ROWS * ldp;
    cp_async_wait_all();
    __syncthreads();
    if (!last) load_rows(u + step, slot ^ 1);
    if (has_l2l) {
      double acc[RB][2];
      unit_gemm(t, Lp, ldp, st.M, ncb, ncb, acc);
      unit_sum(t, acc, sm.part);
      unit_each(t, acc, [&](int r, int c, double a, double b) {
        double2 *o = reinterpret_cast<double2 *>(P + r * ldp + c);
        const double2 w = *o;
        *o = make_double2(w.x + a, w.y + b);
      });
      __syncthreads();
    }
    if (last && threadIdx.x == 0) next_ops();
    c2e_rows_smem<RB>(st.U, st.V, st.sinv, np, P, T, sm.part, sm.orow[slot]);
  }
}

__global__ void __launch_bounds__(NT, 2) k_down_levels(LevelSpans sp, int np, int n_rhs,
                                                    const int *__restrict__ rg,
                                                    const int *__restrict__ parent,
                                                    const LevelOpsDev *__restrict__ ops,
                                                    const double *__restrict__ ple, double *loc,
                                                    int64_t cstride, RadixSync *sync, int *fail) {
  extern __shared__ __align__(16) double smem[];
  __shared__ __align__(16) LevelSmem sm;
  const LevelStage st = level_stage(smem, np, 1, sm.bar);
  double *rows = smem + level_ops_doubles(np, 1);
  auto next_of = [&](int i) {  // the first level from i on in which this block has a tile
    while (i < sp.n && (int64_t)sp.lv[i].tiles * n_rhs <= blockIdx.x / 4) ++i;
    return i;
  };
  int nxt = next_of(0);
  uint32_t fills = 0;
  auto load_m = [&] {  // class c of the parents' L2L operator: its column blocks of each k pair
    if (nxt >= sp.n) return;
    const bool has = sp.m0 + nxt >= 3;
    const uint32_t seg = 64u * np;  // bytes of a k pair's class block
    bulk_expect(sm.bar, has ? seg * (np / 8) : 0u);
    if (!has) return;
    const double2 *src = ops[sp.m0 + nxt - 1].l2l_f + (blockIdx.x & 3) * 4 * np;
    for (int kp = 0; kp < np / 8; ++kp)
      bulk_copy(st.M + kp * 4 * np, src + (size_t)kp * 16 * np, seg, sm.bar);
  };
  if (threadIdx.x == 0 && nxt < sp.n) {
    load_m();
    st.load_uv(ops[sp.m0 + nxt]);
  }
  for (int i = 0; i < sp.n; ++i) {
    const LevelSpan lv = sp.lv[i];
    if (i == nxt) {
      const bool has_l2l = sp.m0 + i >= 3;
      nxt = next_of(i + 1);
      if (!__syncthreads_and(st.wait(fills++))) {
        if (threadIdx.x == 0) atomicExch(fail, 1);
        return;
      }
      if (lv.rb == 1)
        down_level<1>(st, lv, n_rhs, has_l2l, rg, parent, ple, loc, cstride, rows, sm, load_m);
      else
        down_level<2>(st, lv, n_rhs, has_l2l, rg, parent, ple, loc, cstride, rows, sm, load_m);
      if (nxt < sp.n) {
        __syncthreads();  // U and VH have been read
        if (threadIdx.x == 0) st.load_uv(ops[sp.m0 + nxt]);
      }
    }
    if (i + 1 < sp.n && !grid_barrier(sync, fail)) {
      if (nxt < sp.n) st.wait(fills);  // the copies in flight
      return;
    }
  }
}

// Blocks per SM of a level kernel and its most row blocks per tile.  Several
// charge columns fill the SMs by themselves: two blocks where their buffers
// fit with two row blocks each (np <= 40; 16 columns on a ring of 100k: 5319 ->
// 4883 us a step).  A single column's levels run beside the near field, which
// wants the rest of the SM (two blocks there: 779 -> 819 us a product at 250k).
struct LevelFit {
  int per_sm, rb_max;
};
template <class F>
LevelFit level_fit(F &&bytes, int n_rhs) {
  const size_t extra = sizeof(LevelSmem) + 1024 + 64, all = smem_optin() + 1024;
  if (n_rhs > 1 && 2 * (bytes(2) + extra) <= all) return {2, 2};
  int rb = LEVEL_RB;
  while (rb > 1 && bytes(rb) + extra > all) rb /= 2;
  return {1, rb};
}

// ------------------------------------------------------------ evaluation ----
// Work items of a leaf's targets [b, e), for a warp's 32 nodes (any of them
// empty): their chunk counts are summed over the warp and one atomic finds the
// place of all its items, so the list needs no scan of its own.  The warps'
// items follow one another in any order: no item depends on another.
__device__ __forceinline__ void emit_items(int g, int L, const int *__restrict__ off, int b, int e,
                                           bool binned, int4 *__restrict__ items, int *n_items) {
  const int n = (e - b + TCH - 1) / TCH;
  const int at = warp_place(n, n_items);
  if (n == 0) return;
  const int y = level_of_node(off, L, g) | (binned && n > 1 ? EVAL_MULTI : 0) |
                (binned && e - b > 32 ? EVAL_UNORDERED : 0);
  for (int c = 0; c < n; ++c) {
    const int t0 = b + c * TCH;
    items[at + c] = make_int4(g, y, t0, min(TCH, e - t0));
  }
}

// targets sorted by key: each leaf's range by two searches
__global__ void k_items_sorted(int total, int L, const int *__restrict__ off,
                               const uint64_t *__restrict__ code, const uint8_t *__restrict__ flags,
                               const uint64_t *__restrict__ tkeys, int64_t m,
                               int4 *__restrict__ items, int *n_items) {
  const int stride = gridDim.x * blockDim.x;
  for (int g0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); g0 < total; g0 += stride) {
    const int g = g0 + (threadIdx.x & 31);
    int b = 0, e = 0;
    if (g < total && (flags[g] & NF_LEAF) && m > 0) {
      // both ends of the leaf's key range: two branchless lower-bound
      // searches over [0, m) in step (same length, same step count), so each
      // step's two loads are issued together
      const int sh = 2 * (MAXD - level_of_node(off, L, g));
      const uint64_t c = code[g];
      const uint64_t vlo = c << sh, vhi = (c + 1) << sh;
      int64_t b0 = 0, b1 = 0, len = m;
      while (len > 1) {
        const int64_t half = len >> 1;
        const uint64_t k0 = __ldg(tkeys + b0 + half), k1 = __ldg(tkeys + b1 + half);
        b0 += k0 < vlo ? half : 0;
        b1 += k1 < vhi ? half : 0;
        len -= half;
      }
      b = int(b0 + (__ldg(tkeys + b0) < vlo ? 1 : 0));
      e = int(b1 + (__ldg(tkeys + b1) < vhi ? 1 : 0));
    }
    emit_items(g, L, off, b, e, false, items, n_items);
  }
}

// the tree's own sources: each leaf's range is its [bot, top) (the same
// lower-bound searches of the same sorted keys, done by the node pass)
__global__ void k_items_sources(int total, int L, const int *__restrict__ off,
                                const uint8_t *__restrict__ flags, const int *__restrict__ bot,
                                const int *__restrict__ top, int4 *__restrict__ items,
                                int *n_items) {
  const int stride = gridDim.x * blockDim.x;
  for (int g0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); g0 < total; g0 += stride) {
    const int g = g0 + (threadIdx.x & 31);
    const bool leaf = g < total && (flags[g] & NF_LEAF);
    emit_items(g, L, off, leaf ? bot[g] : 0, leaf ? top[g] : 0, false, items, n_items);
  }
}

// binned targets: count[g] of them in leaf g; their places (first[g] on) are
// given out the same way as the items'
__global__ void k_items_binned(int total, int L, const int *__restrict__ off,
                               const int *__restrict__ count, int *__restrict__ first, int *placed,
                               int4 *__restrict__ items, int *n_items) {
  const int stride = gridDim.x * blockDim.x;
  for (int g0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); g0 < total; g0 += stride) {
    const int g = g0 + (threadIdx.x & 31);
    const int n = g < total ? count[g] : 0;
    const int b = warp_place(n, placed);
    if (g < total) first[g] = b;
    emit_items(g, L, off, b, b + n, true, items, n_items);
  }
}

// KIFMM evaluation of an item: L2T (flexmm/flexmm2d/kifmm.py:106-120: the
// leaf's equivalent sources on its large circle, swept like any other
// sources) and P2P.
// PART: EVAL_FULL (L2T + P2P), EVAL_NEAR (P2P only, into near[], caller's
// point order) or EVAL_FAR (L2T only, plus near[]: out = far + near).
template <class KF, int NOUT, int PART, bool DIP = false, bool CAT = false>
struct KIPolicy : ChargePolicy<KF, NOUT, DIP, CAT> {
  using Base = ChargePolicy<KF, NOUT, DIP, CAT>;
  static_assert(PART == EVAL_FULL || NOUT == 1, "split evaluation: potential only");
  static_assert(!CAT || PART == EVAL_NEAR, "categories: near field only");
  static constexpr bool kNear = PART != EVAL_FAR, kFar = PART != EVAL_NEAR;
  static constexpr int SMAX = Base::SMAX;
  struct FarSmem {
    double2 xy[64];
    double q[64];
    double cx, cy;
  };
  struct NoSmem {
    FunctorSmem<KF> f;
  };
  struct Smem : std::conditional<kNear, typename Base::Smem, NoSmem>::type {
    typename std::conditional<kFar, FarSmem, char>::type far;
  };
  int neq, np;
  const double *xmid, *ymid, *loc;
  const LevelOpsDev *ops;
  double *near;
  const int *fail;  // PassArgs::fail

  // (the near field alone reads no expansions, and runs beside the passes)
  __device__ __forceinline__ bool failed() const { return kFar && fail && *fail; }
  __device__ __forceinline__ void stage_far(Smem &sm, int g, int lev) const {
    if constexpr (kFar) {
      for (int k = threadIdx.x; k < neq; k += EV_THREADS) {
        sm.far.q[k] = loc[(size_t)g * np + k] * Base::fold();
        sm.far.xy[k] = make_double2(ops[lev].lx[k], ops[lev].ly[k]);
      }
      if (threadIdx.x == 64) {
        sm.far.cx = xmid[g];
        sm.far.cy = ymid[g];
      }
    }
  }
  __device__ __forceinline__ void stage(Smem &sm, int i, int j) const {
    if constexpr (kNear) Base::stage(sm, i, j);
  }
  template <int R>
  __device__ __forceinline__ void sweep(const KF &K, const Smem &sm, const double (&x)[R],
                                        const double (&y)[R],
                                        const typename Base::template Tgt<R> &tg, int lo, int hi,
                                        int G, double (&v)[R][Base::NV]) const {
    if constexpr (kNear) Base::template sweep<R>(K, sm, x, y, tg, lo, hi, G, v);
  }
  template <int R>
  __device__ __forceinline__ void far_field(const KF &K, const Smem &sm, int, int,
                                            const double (&x)[R], const double (&y)[R], int warp,
                                            int sub, int G, double (&v)[R][Base::NV]) const {
    if constexpr (kFar) {
      double dx[R], dy[R];
      long long none[R] = {};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        dx[r] = x[r] - sm.far.cx;
        dy[r] = y[r] - sm.far.cy;
      }
      const int lo = (neq * warp) / EV_WARPS + sub, hi = (neq * (warp + 1)) / EV_WARPS;
      if constexpr (NOUT == 1)
        pot_sweep<KF, R, false, false>(K, sm.far.xy, sm.far.q, nullptr, nullptr, dx, dy, none, lo,
                                       hi, G, 0, v);
      else
        grad_sweep<KF, R>(K, sm.far.xy, sm.far.q, dx, dy, lo, hi, G, 0, v);
    }
  }
  __device__ __forceinline__ void store(int i, const double (&o)[NOUT]) const {
    if constexpr (PART == EVAL_NEAR)
      near[i] = o[0];
    else if constexpr (PART == EVAL_FAR)
      this->out[i] = o[0] + near[i];
    else
      Base::store(i, o);
  }
};

// the policy's fields that every part has
template <class Pol>
Pol ki_policy(const PassArgs &a, const double *tau_s, const double *loc, int check, double *out,
              int64_t ld_out, double *near) {
  const TreeDev &td = *a.td;
  Pol p{};
  p.kp = a.kp;
  p.sx = td.sx.get();
  p.sy = td.sy.get();
  p.tau = tau_s;
  p.dvx = a.dvx;
  p.dvy = a.dvy;
  p.check = check;
  p.out = out;
  p.ld_out = ld_out;
  p.neq = a.neq;
  p.np = a.np;
  p.xmid = td.xmid.get();
  p.ymid = td.ymid.get();
  p.loc = loc;
  p.ops = a.ops_dev;
  p.near = near;
  p.fail = a.fail;
  return p;
}

ItemArgs item_args(const PassArgs &a, const int4 *items, int *n_items, int counter,
                   const double *txs, const double *tys, const int *tperm) {
  const TreeDev &td = *a.td;
  return ItemArgs{items, n_items, n_items + 1 + counter, td.coll.get(), td.bot.get(),
                  td.top.get(), txs, tys, tperm};
}

// resident blocks per SM the potential and gradient evaluations are built for
constexpr int EVAL_BLOCKS = 8, EVAL_BLOCKS_GRAD = 6;

template <class Pol, int BLOCKS>
void launch_items(const Pol &pol, const ItemArgs &ia, int64_t units, int per_sm, cudaStream_t s) {
  k_items<Pol, BLOCKS><<<work_grid(units, per_sm), EV_THREADS, 0, s>>>(pol, ia);
  FMMB_CUDA(cudaGetLastError());
}

// Several charge columns on one tree (multi-RHS): columns r0 .. r0 + R - 1
// of the charges (stride n_src) and locals (stride col_stride); each kernel
// value (L2T and P2P) is computed once and applied to the R columns.  Output
// row r of out (stride ld_out).  One work item = (leaf, up to 128 targets);
// the leaf's equivalent sources are staged and swept as its neighbours are.
// Bound by the kernel values and the columns' FMAs, whose charges are read from
// shared memory two at a time.  16 columns of K0 at 60k points on a ring:
// 541 us in two launches of 8 columns before, 312 in one.
constexpr int SMAX_MR = 192;
template <class KF, int R>
__global__ void __launch_bounds__(TCH) k_evaluate_multi(KernelParams kp, int neq, int np, int ncol,
                                                        const int4 *__restrict__ items,
                                                        const int *__restrict__ n_items_ptr,
                                                        const int *__restrict__ coll,
                                                        const int *__restrict__ bot,
                                                        const int *__restrict__ top,
                                                        const double *__restrict__ xmid,
                                                        const double *__restrict__ ymid,
                                                        const double *__restrict__ sx,
                                                        const double *__restrict__ sy,
                                                        const double *__restrict__ tau, int64_t n_src,
                                                        const LevelOpsDev *__restrict__ ops,
                                                        const double *__restrict__ loc,
                                                        int64_t col_stride,
                                                        const double *__restrict__ txs,
                                                        const double *__restrict__ tys,
                                                        const int *__restrict__ tperm, int check,
                                                        double *__restrict__ out, int64_t ld_out,
                                                        const int *__restrict__ fail) {
  __shared__ double2 sxy[SMAX_MR];
  __shared__ __align__(16) double stau[SMAX_MR][R + 2];  // (padded: fewer bank conflicts)
  __shared__ int rb[9], rs[10];
  __shared__ double red[R][TCH / 32];
  __shared__ FunctorSmem<KF> fsm;
  KF K(kp);
  fsm.bind(K);
  const int n_items = *n_items_ptr;
  const bool failed = fail && *fail;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int4 it = items[item];
    const int g = it.x, lev = it.y & EVAL_LEVEL_MASK, t0 = it.z, cnt = it.w;
    int G = 1;
    if (!(it.y & EVAL_MULTI))
      while (2 * G * cnt <= TCH) G *= 2;
    const int t = threadIdx.x / G, sub = threadIdx.x % G;
    const bool valid = t < cnt;
    const double x = valid ? txs[t0 + t] : 0.0, y = valid ? tys[t0 + t] : 0.0;
    if (threadIdx.x < 9) {
      const int cg = coll[(size_t)g * 9 + threadIdx.x];
      rb[threadIdx.x] = cg >= 0 ? bot[cg] : 0;
      rs[threadIdx.x + 1] = cg >= 0 ? top[cg] - bot[cg] : 0;
    }
    if (threadIdx.x == 0) rs[0] = 0;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int c = 1; c <= 9; ++c) rs[c] += rs[c - 1];
    double u[R];
#pragma unroll
    for (int c = 0; c < R; ++c) u[c] = 0.0;
    auto sweep = [&](int n, double px, double py, bool chk) {  // the staged sources
      if (!valid) return;
#pragma unroll 2
      for (int j = sub; j < n; j += G) {
        const double2 q = sxy[j];
        if (chk && px - q.x == 0.0 && py - q.y == 0.0) continue;
        const double kv = K(q.x, q.y, px, py);
        const double2 *tq = reinterpret_cast<const double2 *>(stau[j]);
#pragma unroll
        for (int c = 0; c < R / 2; ++c) {
          const double2 w = tq[c];
          u[2 * c] = fma(kv, w.x, u[2 * c]);
          u[2 * c + 1] = fma(kv, w.y, u[2 * c + 1]);
        }
      }
    };
    if (lev >= 2) {  // L2T
      for (int k = threadIdx.x; k < neq; k += TCH) sxy[k] = make_double2(ops[lev].lx[k], ops[lev].ly[k]);
      for (int i = threadIdx.x; i < neq * R; i += TCH) {
        const int c = i / neq, k = i - c * neq;
        stau[k][c] = c < ncol ? loc[c * col_stride + (size_t)g * np + k] : 0.0;
      }
      __syncthreads();
      sweep(neq, x - xmid[g], y - ymid[g], false);
    }
    __syncthreads();
    const int ns = rs[9];
    for (int base = 0; base < ns; base += SMAX_MR) {
      const int nb = min(SMAX_MR, ns - base);
      for (int i = threadIdx.x; i < nb; i += TCH) {
        const int idx = base + i;
        int c = 0;
        while (idx >= rs[c + 1]) ++c;
        const int j = rb[c] + (idx - rs[c]);
        sxy[i] = make_double2(sx[j], sy[j]);
#pragma unroll
        for (int q = 0; q < R; ++q) stau[i][q] = q < ncol ? tau[q * n_src + j] : 0.0;
      }
      __syncthreads();
      sweep(nb, x, y, check);
      __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < R; ++c) {
      double w = u[c];
      for (int q = min(G, 32) >> 1; q >= 1; q >>= 1) w += __shfl_xor_sync(0xffffffffu, w, q);
      if (G > 32) {
        if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = w;
        __syncthreads();
        if (sub == 0) {
          w = 0.0;
          for (int q = 0; q < G / 32; ++q) w += red[c][(threadIdx.x >> 5) + q];
        }
      }
      if (valid && sub == 0 && c < ncol) out[c * ld_out + tperm[t0 + t]] = failed ? nan("") : w;
    }
    __syncthreads();
  }
}

// FP64 direct sum (kernel_apply / kernel_apply_single_check,
// flexmm/flexmm2d/helpers.py:91-116): all sources, one target per thread,
// sources staged through shared memory
template <class KF>
__global__ void __launch_bounds__(256) k_direct(KernelParams kp, const double *__restrict__ sx,
                                                const double *__restrict__ sy,
                                                const double *__restrict__ tau, int64_t ns,
                                                const double *__restrict__ tx,
                                                const double *__restrict__ ty, int64_t nt,
                                                int check, double *__restrict__ out) {
  __shared__ double qx[256], qy[256], qt[256];
  const KF K(kp);
  for (int64_t base = (int64_t)blockIdx.x * 256; base < nt; base += (int64_t)gridDim.x * 256) {
    const int64_t i = base + threadIdx.x;
    const bool valid = i < nt;
    const double x = valid ? tx[i] : 0.0, y = valid ? ty[i] : 0.0;
    double u = 0.0;
    for (int64_t j0 = 0; j0 < ns; j0 += 256) {
      const int nj = (int)(ns - j0 < 256 ? ns - j0 : 256);
      __syncthreads();
      if (threadIdx.x < nj) {
        qx[threadIdx.x] = sx[j0 + threadIdx.x];
        qy[threadIdx.x] = sy[j0 + threadIdx.x];
        qt[threadIdx.x] = tau[j0 + threadIdx.x];
      }
      __syncthreads();
      if (valid)
        for (int j = 0; j < nj; ++j) {
          if (check && x - qx[j] == 0.0 && y - qy[j] == 0.0) continue;
          u = fma(K(qx[j], qy[j], x, y), qt[j], u);
        }
    }
    if (valid) out[i] = u;
  }
}

__global__ void k_gather_sorted(const double *__restrict__ v, const int *__restrict__ perm,
                                int64_t n, double *__restrict__ o, int64_t ld_v) {
  v += blockIdx.y * ld_v;  // column blockIdx.y
  o += blockIdx.y * n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    o[i] = v[perm[i]];
}

template <class KF>
void upward_impl(const PassArgs &a, const double *tau_s, double *mult, cudaStream_t s, int n_rhs,
                 int64_t tstride, int64_t cstride) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  const int np = a.np;
  if (th.L < 3) return;
  PhaseTimer timer(PH_UPWARD, s);
  const int per_sm = 8;
  const int64_t warps = std::min<int64_t>(th.n_total(), (int64_t)148 * per_sm * S2M_WARPS);
  const int s2m_grid = int((warps + S2M_WARPS - 1) / S2M_WARPS);
  if (n_rhs > 1) {
    k_s2m_multi<KF><<<dim3(s2m_grid, (n_rhs + S2M_COLS - 1) / S2M_COLS), 32 * S2M_WARPS, 0, s>>>(
        a.kp, a.neq, np, th.L, td.dev_off.get(), td.uplist.get(), td.n_up.get(), td.bot.get(),
        td.top.get(), td.xmid.get(), td.ymid.get(), td.sx.get(), td.sy.get(), tau_s, a.ops_dev, mult,
        n_rhs, tstride, cstride);
  } else {
    auto launch = [&](auto kern) {
      kern<<<s2m_grid, 32 * S2M_WARPS, 0, s>>>(
          a.kp, a.neq, np, th.L, td.dev_off.get(), td.uplist.get(), td.n_up.get(), td.bot.get(),
          td.top.get(), td.xmid.get(), td.ymid.get(), td.sx.get(), td.sy.get(), tau_s, a.ops_dev,
          mult, a.dvx, a.dvy);
    };
    if (!a.dvx)
      launch(k_s2m<KF, false>);
    else if constexpr (std::is_same<KF, LaplaceF64T>::value)
      launch(k_s2m<KF, true>);
    else
      throw Error(ERR_UNSUPPORTED, "dipole sources: Laplace kernel only");
  }
  FMMB_CUDA(cudaGetLastError());
  const size_t c2e_bytes = c2e_leaves_smem(np);
  smem_limit(k_c2e_leaves, c2e_bytes);
  // at least two tiles a block: its operators serve 32 rows or more
  const int64_t c2e_tiles = (int64_t)n_rhs * ((th.n_total() + C2E_ROWS - 1) / C2E_ROWS);
  k_c2e_leaves<<<work_grid((c2e_tiles + 1) / 2, 2), NT, c2e_bytes, s>>>(
      np, th.L, n_rhs, td.dev_off.get(), td.uplist.get(), td.n_up.get(), a.ops_dev, mult, cstride);
  FMMB_CUDA(cudaGetLastError());
  LevelSpans sp{};
  sp.m0 = th.L - 2;
  const LevelFit fit = level_fit([&](int rb) { return up_smem(np, rb); }, n_rhs);
  const int rb_max = fit.rb_max;
  const size_t up_bytes = up_smem(np, rb_max);
  smem_limit(k_up_levels, up_bytes);
  const int64_t cap = coop_blocks((const void *)k_up_levels, NT, up_bytes, fit.per_sm);
  int64_t widest = 0;
  for (int m = th.L - 2; m >= 2; --m) {
    const int n_groups = (th.off[m + 2] - th.off[m + 1]) / 4;
    const int64_t units = (int64_t)((n_groups + 7) / 8) * n_rhs;
    const int rb = level_rows(units, cap, rb_max);
    LevelSpan &lv = sp.lv[sp.n++];
    lv = LevelSpan{th.off[m + 1], n_groups, rb, (n_groups + 8 * rb - 1) / (8 * rb)};
    widest = std::max<int64_t>(widest, (int64_t)lv.tiles * n_rhs);
  }
  if (widest == 0) return;
  const int grid = int(std::min(widest, cap));
  int n_rhs_ = n_rhs, np_ = np;
  const int *parent = td.parent.get();
  const LevelOpsDev *ops = a.ops_dev;
  RadixSync *sync = a.sync;
  int *fail = a.fail;
  void *args[] = {&sp, &np_, &n_rhs_, &parent, &ops, &mult, &cstride, &sync, &fail};
  launch_coop(reinterpret_cast<const void *>(k_up_levels), grid, NT, args, up_bytes, s);
}

}  // namespace

namespace {
// the list of targets sorted by key, or of the tree's own sources
void items_sorted(const PassArgs &a, const uint64_t *tkeys, int64_t m, int4 *items, int *n_items,
                  cudaStream_t s) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  const int total = th.n_total(), grid = grid_for(total, 256);
  FMMB_CUDA(cudaMemsetAsync(n_items, 0, (1 + EVAL_COUNTERS) * sizeof(int), s));
  if (tkeys == td.pkeys.get() && m == th.n_points)
    k_items_sources<<<grid, 256, 0, s>>>(total, th.L, td.dev_off.get(), td.flags.get(),
                                         td.bot.get(), td.top.get(), items, n_items);
  else
    k_items_sorted<<<grid, 256, 0, s>>>(total, th.L, td.dev_off.get(), td.code.get(),
                                        td.flags.get(), tkeys, m, items, n_items);
  FMMB_CUDA(cudaGetLastError());
}
}  // namespace

void eval_items(const PassArgs &a, const uint64_t *tkeys, int64_t m, EvalItems &it, cudaStream_t s) {
  it.items.alloc(a.th->n_total() + m / TCH + 1, s);
  it.n_items.alloc(1 + EVAL_COUNTERS, s);
  items_sorted(a, tkeys, m, it.items.get(), it.n_items.get(), s);
}

void eval_items_binned(const PassArgs &a, const double *tx, const double *ty, int64_t m,
                       EvalItems &it, double *txs, double *tys, int *tperm, cudaStream_t s) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  const int total = th.n_total();
  DevBuf<int> first, leaf_of, slot;
  first.alloc(total, s);
  leaf_of.alloc(m, s);
  slot.alloc(m, s);
  it.items.alloc(total + m / TCH + 1, s);
  // the list's counters, the targets placed so far and the nodes' counts: one memset
  it.n_items.alloc(2 + EVAL_COUNTERS + total, s);
  it.n_items.zero(s);
  int *placed = it.n_items.get() + 1 + EVAL_COUNTERS, *count = placed + 1;
  bin_points(tx, ty, m, td, th, count, leaf_of.get(), slot.get(), s);
  k_items_binned<<<grid_for(total, 256), 256, 0, s>>>(total, th.L, td.dev_off.get(), count,
                                                      first.get(), placed, it.items.get(),
                                                      it.n_items.get());
  FMMB_CUDA(cudaGetLastError());
  scatter_binned(tx, ty, m, leaf_of.get(), slot.get(), first.get(), txs, tys, tperm, s);
}

namespace {
template <class KF>
void evaluate_impl(const PassArgs &a, const double *tau_s, const double *loc, const double *txs,
                   const double *tys, const uint64_t *tkeys, const int *tperm, int64_t m, int check,
                   int nout, double *out, int64_t ld_out, cudaStream_t s, const EvalItems *pre) {
  EvalItems own;
  if (!pre) eval_items(a, tkeys, m, own, s);
  const EvalItems &it = pre ? *pre : own;
  const int64_t units = a.th->n_total() + m / TCH + 1;  // work items, upper bound
  PhaseTimer timer(PH_EVAL, s);
  const ItemArgs ia = item_args(a, it.items.get(), it.n_items.get(), 0, txs, tys, tperm);
  if (a.dvx) {
    FMMB_CHECK(nout == 1, ERR_UNSUPPORTED, "dipole sources: potential only");
    if constexpr (std::is_same<KF, LaplaceF64T>::value) {
      using Pol = KIPolicy<KF, 1, EVAL_FULL, true>;
      launch_items<Pol, EVAL_BLOCKS_GRAD>(
          ki_policy<Pol>(a, tau_s, loc, check, out, ld_out, nullptr), ia, units, EVAL_BLOCKS_GRAD, s);
    } else {
      throw Error(ERR_UNSUPPORTED, "dipole sources: Laplace kernel only");
    }
  } else if (nout == 3) {
    using Pol = KIPolicy<KF, 3, EVAL_FULL>;
    launch_items<Pol, EVAL_BLOCKS_GRAD>(ki_policy<Pol>(a, tau_s, loc, check, out, ld_out, nullptr),
                                        ia, units, EVAL_BLOCKS_GRAD, s);
  } else {
    using Pol = KIPolicy<KF, 1, EVAL_FULL>;
    launch_items<Pol, EVAL_BLOCKS>(ki_policy<Pol>(a, tau_s, loc, check, out, ld_out, nullptr), ia,
                                   units, EVAL_BLOCKS, s);
  }
}
}  // namespace

void run_upward(const PassArgs &a, const double *tau_s, double *mult, cudaStream_t s, int n_rhs,
                int64_t tstride, int64_t cstride) {
  FMMB_CHECK(n_rhs >= 1 && n_rhs <= 65535, ERR_INVALID_ARGUMENT, "1..65535 charge columns");
  switch (a.kernel_id) {
    case KERNEL_LAPLACE: upward_impl<LaplaceF64T>(a, tau_s, mult, s, n_rhs, tstride, cstride); break;
    case KERNEL_MOD_HELMHOLTZ:
      upward_impl<ModHelmholtzF64T>(a, tau_s, mult, s, n_rhs, tstride, cstride);
      break;
    case KERNEL_RADIAL_TABLE:
      upward_impl<RadialTableF64>(a, tau_s, mult, s, n_rhs, tstride, cstride);
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
}

// targets (times charge columns) below which M2L tiles hold 16 targets: fewer
// would leave SMs without one of 64 (3k points: 45 us with tiles of 64, 24 now)
constexpr int64_t M2L_FEW_TARGETS = 148 * 64;

void run_m2l(const PassArgs &a, const double *mult, double *ple, cudaStream_t s, int n_rhs,
             int64_t cstride) {
  const TreeHost &th = *a.th;
  if (th.L < 3) return;
  FMMB_CHECK(th.L <= FMM_MAX_LEVELS_DEV, ERR_INVALID_ARGUMENT, "too many levels");
  int64_t targets = 0;
  for (int m = 2; m < th.L; ++m) targets += 4 * (int64_t)(th.rg_hi[m] - th.rg_lo[m]);
  // few targets: smaller tiles, for more blocks and a shorter chain in each
  const int tt = targets * n_rhs < M2L_FEW_TARGETS ? 16 : a.np <= 32 || a.np > 64 ? 32 : 64;
  M2LTiles tl{};
  tl.n_levels = th.L;
  int tiles = 0;
  for (int m = 0; m < th.L; ++m) {
    tl.rg_lo[m] = th.rg_lo[m];
    tl.rg_cnt[m] = th.rg_hi[m] - th.rg_lo[m];
    for (int c = 0; c < 4; ++c) {
      tl.tile_start[4 * m + c] = tiles;
      if (m >= 2) tiles += (tl.rg_cnt[m] + tt - 1) / tt;
    }
  }
  tl.tile_start[4 * th.L] = tiles;
  if (tiles == 0) return;
  PhaseTimer timer(PH_M2L, s);
  auto launch = [&](auto ncb) {
    constexpr int NCB = decltype(ncb)::value;
    const size_t sm = M2LShape<NCB>::smem(tt);
    static_assert(M2LShape<NCB>::kTargets == (NCB <= 4 || NCB > 8 ? 32 : 64), "tiles are counted for this size");
    smem_limit(k_m2l<NCB>, M2LShape<NCB>::smem(M2LShape<NCB>::kTargets));
    k_m2l<NCB><<<dim3(tiles, n_rhs), 32 * NCB, sm, s>>>(tl, tt, a.td->rg.get(), a.td->il.get(),
                                                        a.ops_dev, mult, ple, cstride);
    FMMB_CUDA(cudaGetLastError());
  };
  switch (a.np / 8) {
    case 1: launch(std::integral_constant<int, 1>{}); break;
    case 2: launch(std::integral_constant<int, 2>{}); break;
    case 3: launch(std::integral_constant<int, 3>{}); break;
    case 4: launch(std::integral_constant<int, 4>{}); break;
    case 5: launch(std::integral_constant<int, 5>{}); break;
    case 6: launch(std::integral_constant<int, 6>{}); break;
    case 7: launch(std::integral_constant<int, 7>{}); break;
    case 8: launch(std::integral_constant<int, 8>{}); break;
    case 9: launch(std::integral_constant<int, 9>{}); break;  // Stokes, Nequiv 28-35
    default: throw Error(ERR_UNSUPPORTED, "unexpected operator size");
  }
}

void run_downward(const PassArgs &a, const double *ple, double *loc, cudaStream_t s, int n_rhs,
                  int64_t cstride) {
  const TreeHost &th = *a.th;
  const TreeDev &td = *a.td;
  LevelSpans sp{};
  sp.m0 = 2;
  const LevelFit fit = level_fit([&](int rb) { return down_smem(a.np, rb); }, n_rhs);
  const int rb_max = fit.rb_max;
  const size_t bytes = down_smem(a.np, rb_max);
  smem_limit(k_down_levels, bytes);
  const int64_t cap = coop_blocks((const void *)k_down_levels, NT, bytes, fit.per_sm) / 4 * 4;
  FMMB_CHECK(cap >= 4, ERR_UNSUPPORTED, "the downward pass needs four SMs");
  int64_t widest = 0;
  for (int m = 2; m < th.L; ++m) {
    const int lo = th.rg_lo[m], cnt = std::max(0, th.rg_hi[m] - th.rg_lo[m]);
    const int64_t units = (int64_t)((cnt + 7) / 8) * n_rhs;
    const int rb = level_rows(units, cap / 4, rb_max);
    LevelSpan &lv = sp.lv[sp.n++];
    lv = LevelSpan{lo, cnt, rb, (cnt + 8 * rb - 1) / (8 * rb)};
    widest = std::max<int64_t>(widest, 4 * (int64_t)lv.tiles * n_rhs);
  }
  if (widest == 0) return;
  const int grid = int(std::min(widest, cap));
  PhaseTimer timer(PH_DOWNWARD, s);
  int n_rhs_ = n_rhs, np_ = a.np;
  const int *rg = td.rg.get(), *parent = td.parent.get();
  const LevelOpsDev *ops = a.ops_dev;
  RadixSync *sync = a.sync + 1;
  int *fail = a.fail;
  void *args[] = {&sp, &np_, &n_rhs_, &rg, &parent, &ops, &ple, &loc, &cstride, &sync, &fail};
  launch_coop(reinterpret_cast<const void *>(k_down_levels), grid, NT, args, bytes, s);
}

void run_evaluate(const PassArgs &a, const double *tau_s, const double *loc, const double *txs,
                  const double *tys, const uint64_t *tkeys, const int *tperm, int64_t m, int check,
                  int nout, double *out, int64_t ld_out, cudaStream_t s, const EvalItems *pre) {
  if (m == 0) return;
  switch (a.kernel_id) {
    case KERNEL_LAPLACE:
      evaluate_impl<LaplaceF64T>(a, tau_s, loc, txs, tys, tkeys, tperm, m, check, nout, out, ld_out,
                                 s, pre);
      break;
    case KERNEL_MOD_HELMHOLTZ:
      evaluate_impl<ModHelmholtzF64T>(a, tau_s, loc, txs, tys, tkeys, tperm, m, check, nout, out,
                                     ld_out, s, pre);
      break;
    case KERNEL_RADIAL_TABLE:
      FMMB_CHECK(nout == 1, ERR_UNSUPPORTED, "tabulated kernels evaluate potentials only");
      evaluate_impl<RadialTableF64>(a, tau_s, loc, txs, tys, tkeys, tperm, m, check, nout, out,
                                    ld_out, s, pre);
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
}

namespace {
template <class KF, bool DIP>
void evaluate_split_impl(const PassArgs &a, const double *tau_s, const double *loc, int check,
                         double *out, cudaStream_t s, const SplitEval &se) {
  const TreeDev &td = *a.td;
  const int64_t m = a.th->n_points;
  FMMB_CUDA(cudaStreamWaitEvent(se.side, se.ready, 0));
  SplitScratch own, &w = se.scratch ? *se.scratch : own;
  if (!se.scratch) w.alloc(a.th->n_total(), m, false, se.side);
  EvalItems &it = w.it;
  DevBuf<double> &near = w.near;
  eval_items(a, td.pkeys.get(), m, it, se.side);
  const int64_t units = a.th->n_total() + m / TCH + 1;  // work items, upper bound
  {
    // the SMs keep their largest shared-memory carveout while near-field
    // blocks sit on them, so the level passes' CTAs still fit beside them
    using Near = KIPolicy<KF, 1, EVAL_NEAR, DIP>;
    static const bool carveout_set = [] {
      FMMB_CUDA(cudaFuncSetAttribute(k_items<Near, EVAL_BLOCKS>,
                                     cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
      return true;
    }();
    (void)carveout_set;
    PhaseTimer timer(PH_EVAL, se.side);
    ItemArgs ia = item_args(a, it.items.get(), it.n_items.get(), 0, td.sx.get(), td.sy.get(),
                            td.ordv.get());
    ia.per_block = NEAR_ITEMS_PER_BLOCK;
    const int blocks = int((units + NEAR_ITEMS_PER_BLOCK - 1) / NEAR_ITEMS_PER_BLOCK);
    k_items<Near, EVAL_BLOCKS><<<blocks, EV_THREADS, 0, se.side>>>(
        ki_policy<Near>(a, tau_s, loc, check, out, 0, near.get()), ia);
    FMMB_CUDA(cudaGetLastError());
  }
  FMMB_CUDA(cudaEventRecord(se.near_done, se.side));
  FMMB_CUDA(cudaStreamWaitEvent(s, se.near_done, 0));
  {
    PhaseTimer timer(PH_EVAL, s);
    using Far = KIPolicy<KF, 1, EVAL_FAR>;
    launch_items<Far, EVAL_BLOCKS>(
        ki_policy<Far>(a, tau_s, loc, check, out, 0, near.get()),
        item_args(a, it.items.get(), it.n_items.get(), 1, td.sx.get(), td.sy.get(), td.ordv.get()),
        units, EVAL_BLOCKS, s);
  }
  // the scratch is used again (or freed) on the side stream once the plan
  // stream is done with it
  FMMB_CUDA(cudaEventRecord(se.far_done, s));
  FMMB_CUDA(cudaStreamWaitEvent(se.side, se.far_done, 0));
}

template <class KF>
void evaluate_multi_impl(const PassArgs &a, const double *tau_s, int64_t n_src, int n_rhs,
                         const double *loc, int64_t col_stride, const double *txs,
                         const double *tys, const uint64_t *tkeys, const int *tperm, int64_t m,
                         int check, double *out, int64_t ld_out, cudaStream_t s) {
  const TreeDev &td = *a.td;
  EvalItems it;
  eval_items(a, tkeys, m, it, s);
  PhaseTimer timer(PH_EVAL, s);
  // columns at a time: 16 where there are more than 8 (the kernel values of a
  // second launch cost more than the smaller occupancy)
  for (int r0 = 0; r0 < n_rhs;) {
    auto launch = [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int ncol = std::min(R, n_rhs - r0);
      k_evaluate_multi<KF, R><<<work_grid(a.th->n_total() + m / TCH + 1, 8), TCH, 0, s>>>(
          a.kp, a.neq, a.np, ncol, it.items.get(), it.n_items.get(), td.coll.get(), td.bot.get(),
          td.top.get(), td.xmid.get(), td.ymid.get(), td.sx.get(), td.sy.get(), tau_s + r0 * n_src,
          n_src, a.ops_dev, loc + r0 * col_stride, col_stride, txs, tys, tperm, check,
          out + r0 * ld_out, ld_out, a.fail);
      FMMB_CUDA(cudaGetLastError());
      r0 += R;
    };
    if (n_rhs - r0 > 8)
      launch(std::integral_constant<int, 16>{});
    else
      launch(std::integral_constant<int, 8>{});
  }
}
}  // namespace

void run_evaluate_multi(const PassArgs &a, const double *tau_s, int64_t n_src, int n_rhs,
                        const double *loc, int64_t col_stride, const double *txs, const double *tys,
                        const uint64_t *tkeys, const int *tperm, int64_t m, int check, double *out,
                        int64_t ld_out, cudaStream_t s) {
  if (m == 0 || n_rhs == 0) return;
  switch (a.kernel_id) {
    case KERNEL_LAPLACE:
      evaluate_multi_impl<LaplaceF64T>(a, tau_s, n_src, n_rhs, loc, col_stride, txs, tys, tkeys,
                                      tperm, m, check, out, ld_out, s);
      break;
    case KERNEL_MOD_HELMHOLTZ:
      evaluate_multi_impl<ModHelmholtzF64T>(a, tau_s, n_src, n_rhs, loc, col_stride, txs, tys, tkeys,
                                           tperm, m, check, out, ld_out, s);
      break;
    case KERNEL_RADIAL_TABLE:
      evaluate_multi_impl<RadialTableF64>(a, tau_s, n_src, n_rhs, loc, col_stride, txs, tys, tkeys,
                                          tperm, m, check, out, ld_out, s);
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
}

void run_evaluate_sources_split(const PassArgs &a, const double *tau_s, const double *loc,
                                int check, double *out, cudaStream_t s, const SplitEval &se) {
  if (a.th->n_points == 0) return;
  switch (a.kernel_id) {
    case KERNEL_LAPLACE:
      if (a.dvx)
        evaluate_split_impl<LaplaceF64T, true>(a, tau_s, loc, check, out, s, se);
      else
        evaluate_split_impl<LaplaceF64T, false>(a, tau_s, loc, check, out, s, se);
      break;
    case KERNEL_MOD_HELMHOLTZ:
      FMMB_CHECK(!a.dvx, ERR_UNSUPPORTED, "dipole sources: Laplace kernel only");
      evaluate_split_impl<ModHelmholtzF64T, false>(a, tau_s, loc, check, out, s, se);
      break;
    case KERNEL_RADIAL_TABLE:
      FMMB_CHECK(!a.dvx, ERR_UNSUPPORTED, "dipole sources: Laplace kernel only");
      evaluate_split_impl<RadialTableF64, false>(a, tau_s, loc, check, out, s, se);
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
}

namespace {
template <class KF>
void local_impl(const PassArgs &a, const double *tau_s, const double *txs, const double *tys,
                const uint64_t *tkeys, const int *tperm, int64_t m, int check,
                const int64_t *scat, const int64_t *tcat, double *out, cudaStream_t s) {
  EvalItems it;
  eval_items(a, tkeys, m, it, s);
  const int64_t units = a.th->n_total() + m / TCH + 1;
  const ItemArgs ia = item_args(a, it.items.get(), it.n_items.get(), 0, txs, tys, tperm);
  PhaseTimer timer(PH_EVAL, s);
  if (scat) {
    using Pol = KIPolicy<KF, 1, EVAL_NEAR, false, true>;
    Pol pol = ki_policy<Pol>(a, tau_s, nullptr, check, nullptr, 0, out);
    pol.scat = scat;
    pol.tcat = tcat;
    launch_items<Pol, EVAL_BLOCKS>(pol, ia, units, EVAL_BLOCKS, s);
  } else {
    using Pol = KIPolicy<KF, 1, EVAL_NEAR>;
    launch_items<Pol, EVAL_BLOCKS>(ki_policy<Pol>(a, tau_s, nullptr, check, nullptr, 0, out), ia,
                                   units, EVAL_BLOCKS, s);
  }
}
}  // namespace

void run_local_evaluate(const PassArgs &a, const double *tau_s, const double *txs,
                        const double *tys, const uint64_t *tkeys, const int *tperm, int64_t m,
                        int check, const int64_t *scat, const int64_t *tcat, double *out,
                        cudaStream_t s) {
  if (m == 0) return;
  switch (a.kernel_id) {
    case KERNEL_LAPLACE:
      local_impl<LaplaceF64T>(a, tau_s, txs, tys, tkeys, tperm, m, check, scat, tcat, out, s);
      break;
    case KERNEL_MOD_HELMHOLTZ:
      local_impl<ModHelmholtzF64T>(a, tau_s, txs, tys, tkeys, tperm, m, check, scat, tcat, out, s);
      break;
    case KERNEL_RADIAL_TABLE:
      local_impl<RadialTableF64>(a, tau_s, txs, tys, tkeys, tperm, m, check, scat, tcat, out, s);
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
}

__global__ void k_gather_i64(const int64_t *__restrict__ v, const int *__restrict__ perm, int64_t n,
                             int64_t *__restrict__ o) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    o[i] = v[perm[i]];
}

void gather_sorted_i64(const int64_t *v, const int *perm, int64_t n, int64_t *o, cudaStream_t s) {
  if (n == 0) return;
  k_gather_i64<<<grid_for(n, 256), 256, 0, s>>>(v, perm, n, o);
  FMMB_CUDA(cudaGetLastError());
}

void run_direct(int kernel_id, const KernelParams &kp, const double *sx, const double *sy,
                const double *tau, int64_t ns, const double *tx, const double *ty, int64_t nt,
                int check, double *out, cudaStream_t s) {
  if (nt == 0) return;
  PhaseTimer timer(PH_DIRECT, s);
  const int grid = grid_for(nt, 256, 148 * 64);
  switch (kernel_id) {
    case KERNEL_LAPLACE:
      k_direct<LaplaceF64><<<grid, 256, 0, s>>>(kp, sx, sy, tau, ns, tx, ty, nt, check, out);
      break;
    case KERNEL_MOD_HELMHOLTZ:
      k_direct<ModHelmholtzF64><<<grid, 256, 0, s>>>(kp, sx, sy, tau, ns, tx, ty, nt, check, out);
      break;
    case KERNEL_RADIAL_TABLE:
      k_direct<RadialTableF64><<<grid, 256, 0, s>>>(kp, sx, sy, tau, ns, tx, ty, nt, check, out);
      break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
  FMMB_CUDA(cudaGetLastError());
}

void run_evaluate_scratch(const PassArgs &a, const double *tau_s, const double *loc,
                          const double *txs, const double *tys, const uint64_t *tkeys,
                          const int *tperm, int64_t m, int check, double *out, int4 *items,
                          int *n_items, cudaStream_t s) {
  if (m == 0) return;
  const int total = a.th->n_total();
  items_sorted(a, tkeys, m, items, n_items, s);
  PhaseTimer timer(PH_EVAL, s);
  const ItemArgs ia = item_args(a, items, n_items, 0, txs, tys, tperm);
  auto launch = [&](auto kf) {
    using Pol = KIPolicy<typename decltype(kf)::type, 1, EVAL_FULL>;
    launch_items<Pol, EVAL_BLOCKS>(ki_policy<Pol>(a, tau_s, loc, check, out, 0, nullptr), ia,
                                   total + m / TCH + 1, EVAL_BLOCKS, s);
  };
  switch (a.kernel_id) {
    case KERNEL_LAPLACE: launch(TypeOf<LaplaceF64T>{}); break;
    case KERNEL_MOD_HELMHOLTZ: launch(TypeOf<ModHelmholtzF64T>{}); break;
    case KERNEL_RADIAL_TABLE: launch(TypeOf<RadialTableF64>{}); break;
    default: throw Error(ERR_UNSUPPORTED, "unknown kernel id");
  }
}

namespace {
__global__ void k_diag_log2(const double *__restrict__ x, int64_t n, double *__restrict__ out_tab,
                            double *__restrict__ out_lib) {
  __shared__ FunctorSmem<LaplaceF64T> fsm;
  LaplaceF64T K(KernelParams{});
  fsm.bind(K);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double d = x[i];
    out_tab[i] = log2_tab_rare(d) ? log2(d) : log2_tab(d, K.lt);
    out_lib[i] = log2(d);
  }
}
}  // namespace

void run_diag_log2(const double *x, int64_t n, double *out_tab, double *out_lib, cudaStream_t s) {
  if (n == 0) return;
  k_diag_log2<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(x, n, out_tab, out_lib);
  FMMB_CUDA(cudaGetLastError());
}

void gather_sorted(const double *v, const int *perm, int64_t n, double *o, cudaStream_t s,
                   int columns, int64_t ld_v) {
  if (n == 0) return;
  for (int c = 0; c < columns; c += 65535)
    k_gather_sorted<<<dim3(grid_for(n, 256), std::min(columns - c, 65535)), 256, 0, s>>>(
        v + c * ld_v, perm, n, o + c * n, ld_v);
  FMMB_CUDA(cudaGetLastError());
}

}  // namespace fmmb
