// The evaluation of work items, shared by the FP64 forms (KIFMM, black-box,
// Stokes): an item is one leaf and up to 128 of its targets; a block of four
// warps sums the leaf's far field and its colleagues' sources at them
// (flexmm/flexmm2d/fmm.py:158-176, helpers.py:152-194).
//
// Split of the work inside an item: the warps split the sources (each takes
// a quarter of every staged chunk and of the far field's terms), the lanes
// split the targets.  Each full tile of 32 targets is one target per lane,
// two tiles at a time, so that a staged source is read once for two pairs;
// the last, partial tile of r targets gives each of them G = 32 / r lanes
// (rounded down to a power of two), which split the warp's sources again.
// The four warps' partial sums meet in shared memory.  Against the earlier
// split (128 / targets threads per target over the whole block, items dealt
// out statically) this leaves no lane idle on the first 32 targets of a leaf,
// and the hand-out by a counter evens out the blocks.  Measured (kernel alone,
// before -> after, with the log2 table of kernels.cuh): potentials at 1M
// clustered points and a 1000^2 grid 1.51 -> 0.97 ms, at 250k ring points 0.28
// -> 0.18 ms, gradients at 100k points and a 200^2 grid 0.20 -> 0.12 ms.
// Bound by instruction issue beside the FP64 pipe (about 26 instructions, 13
// of them FP64, per pair).
//
// A policy holds what one form sums: its staged source record, the far field
// and the pair sweep.  All its members run on every thread of the block.
// failed(): the expansions are not to be used (the results are NaN then).
#pragma once
#include <type_traits>

#include "fmm.cuh"

namespace fmmb {
namespace {

constexpr int EV_WARPS = 4, EV_THREADS = 32 * EV_WARPS;
static_assert(EV_THREADS == EVAL_CHUNK, "an item's targets fit the block's threads");

template <class T>
struct TypeOf {
  using type = T;
};

struct ItemArgs {
  const int4 *items;
  const int *n_items;  // device count
  int *next;           // hand-out counter, 0 at launch
  const int *coll, *bot, *top;
  const double *txs, *tys;
  const int *tperm;
  // items a block takes before it ends; the grid times this covers the list
  int per_block = 1 << 30;
};

template <class Pol, int BLOCKS>
__global__ void __launch_bounds__(EV_THREADS, BLOCKS) k_items(const Pol pol, const ItemArgs a) {
  __shared__ typename Pol::Smem sm;
  __shared__ double red[Pol::NOUT][EV_WARPS][EVAL_CHUNK];  // partial sums by warp and target
  __shared__ int rb[9], rs[10];  // colleague range begins and prefix sizes
  __shared__ int s_next;
  typename Pol::Kernel K = pol.bind(sm);
  const int n_items = *a.n_items;
  const bool failed = pol.failed();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int item = blockIdx.x, left = a.per_block;
  while (item < n_items && left-- > 0) {
    const int4 it = a.items[item];
    const int g = it.x, lev = it.y & EVAL_LEVEL_MASK, t0 = it.z, cnt = it.w;
    if (tid == 0) s_next = left > 0 ? int(gridDim.x) + atomicAdd(a.next, 1) : 0;
    if (Pol::kNear && warp == 0) {
      const int cg = lane < 9 ? a.coll[(size_t)g * 9 + lane] : -1;
      const int b = cg >= 0 ? a.bot[cg] : 0, n = cg >= 0 ? a.top[cg] - b : 0;
      int p = n;  // inclusive prefix over the nine colleagues
#pragma unroll
      for (int w = 1; w < 16; w <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, p, w);
        if (lane >= w) p += v;
      }
      if (lane < 9) {
        rb[lane] = b;
        rs[lane + 1] = p;
      }
      if (lane == 0) rs[0] = 0;
    }
    const bool far = Pol::kFar && lev >= 2;  // locals of levels 0-1 are zero
    if (far) pol.stage_far(sm, g, lev);
    __syncthreads();
    const int next = s_next;
    const int ns = Pol::kNear ? rs[9] : 0;
    const bool one_chunk = ns <= Pol::SMAX;
    bool staged = false;
    // R tiles of targets from slot t_base on, G lanes per target (R = 1 when G > 1)
    auto tiles = [&](auto rc, int t_base, int G) {
      constexpr int R = decltype(rc)::value;
      const int sub = lane & (G - 1), slot0 = t_base + lane / G;
      double x[R], y[R];
      double acc[R][Pol::NV];
      typename Pol::template Tgt<R> tg;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int t = t0 + min(slot0 + 32 * r, cnt - 1);  // idle lanes repeat the last target
        x[r] = a.txs[t];
        y[r] = a.tys[t];
        pol.load_target(tg, r, a.tperm, t);
#pragma unroll
        for (int v = 0; v < Pol::NV; ++v) acc[r][v] = 0.0;
      }
      if (far) pol.template far_field<R>(K, sm, g, lev, x, y, warp, sub, G, acc);
      for (int base = 0; base < ns; base += Pol::SMAX) {
        const int nb = min(Pol::SMAX, ns - base);
        if (!one_chunk || !staged) {
          if (staged) __syncthreads();  // the chunk before has been read
          for (int i = tid; i < nb; i += EV_THREADS) {
            const int idx = base + i;
            int c = 0;
#pragma unroll
            for (int k = 1; k < 9; ++k) c += idx >= rs[k];
            pol.stage(sm, i, rb[c] + (idx - rs[c]));
          }
          __syncthreads();
          staged = true;
        }
        pol.template sweep<R>(K, sm, x, y, tg, (nb * warp) / EV_WARPS + sub,
                              (nb * (warp + 1)) / EV_WARPS, G, acc);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double o[Pol::NOUT];
        pol.finish(acc[r], o);
#pragma unroll
        for (int k = 0; k < Pol::NOUT; ++k) {
          if (R == 1)
            for (int w = G >> 1; w >= 1; w >>= 1) o[k] += __shfl_xor_sync(0xffffffffu, o[k], w);
          if (sub == 0 && slot0 + 32 * r < cnt) red[k][warp][slot0 + 32 * r] = o[k];
        }
      }
    };
    int t = 0;
    for (; cnt - t >= 64; t += 64) tiles(std::integral_constant<int, 2>{}, t, 1);
    // a leaf whose targets stand in no particular order (EVAL_UNORDERED)
    // gives every target the same split, whatever its place
    if (cnt - t > 32 && (it.y & EVAL_UNORDERED)) {
      tiles(std::integral_constant<int, 2>{}, t, 1);
      t = cnt;
    }
    if (cnt - t >= 32) {
      tiles(std::integral_constant<int, 1>{}, t, 1);
      t += 32;
    }
    if (cnt > t) {
      int G = 1;
      if (!(it.y & EVAL_UNORDERED))
        while (2 * G * (cnt - t) <= 32) G *= 2;
      tiles(std::integral_constant<int, 1>{}, t, G);
    }
    __syncthreads();
    if (tid < cnt) {
      double o[Pol::NOUT];
#pragma unroll
      for (int k = 0; k < Pol::NOUT; ++k)
        o[k] = failed ? nan("")
                      : (red[k][0][tid] + red[k][1][tid]) + (red[k][2][tid] + red[k][3][tid]);
      pol.store(a.tperm[t0 + tid], o);
    }
    item = next;
  }
}

}  // namespace
}  // namespace fmmb
