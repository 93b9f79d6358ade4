// Prefix sums of the tree build (split counts, parent and node flags) and of
// the charges: one launch, the same result on every run.  The functor F makes
// the items and takes their sums, so what computes the flags and what writes by
// the sums needs no launch of its own (the tree build on 100k points: 31
// launches before, 13 now):
//   T value(int i)             item i (may be asked for twice: the same answer)
//   void fallback(int i)       before the barrier: a valid state should it fail
//   void emit(int i, T pos, T v)  its sum and the item itself
//   void failed()              a barrier wait ran out (one thread of the block)
//   void end()                 all threads of the block, after everything
//
// Tiles of SC_THREADS x ITEMS consecutive elements (tile t on block t mod grid):
//   1. every block sums its tiles (each thread its ITEMS items in order,
//      then the threads in a fixed order) into tsum[t]; with one tile per
//      block the tile stays in registers for step 3;
//   2. a grid barrier; every block scans tsum over all tiles in a fixed
//      order (the same numbers on every block and every run) for its tiles'
//      prefixes;
//   3. each thread scans its items onto the prefix of its thread, warp and
//      tile and emits them.
// For floating point the grouping is fixed by the tile and thread layout,
// so results do not depend on timing.  A barrier wait that runs out sets
// *fail (if given) and leaves the fallback.  One tile runs as one block (no
// barrier).
#pragma once
#include "radix.cuh"

namespace fmmb {
namespace {

constexpr int SC_THREADS = 512;
constexpr int SC_ITEMS = 8;  // items a thread; fewer where the tiles would leave SMs idle
constexpr int SC_FEW = 2;    // (100k points: the split scan 12.8 -> 6.9 us)

// exclusive scan of one value per thread of the block; returns this
// thread's prefix, *total the block's sum (warp shuffles, then the warp
// totals in shared memory; fixed order)
template <class T>
__device__ T sc_block_exclusive(T v, T *total) {
  __shared__ T wsum[SC_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  T ex = __shfl_up_sync(0xffffffffu, incl, 1);  // exclusive, not incl - v (exact for floats)
  if (lane == 0) ex = T(0);
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  T before = T(0), all = T(0);
  for (int q = 0; q < SC_THREADS / 32; ++q) {
    if (q == warp) before = all;
    all += wsum[q];
  }
  __syncthreads();  // wsum reused by the next call
  *total = all;
  return before + ex;
}

template <class T, bool INCLUSIVE, int ITEMS, class F>
__global__ void __launch_bounds__(SC_THREADS, 2)
    k_scan(F f, int n, T *tsum, RadixSync *sync, int *fail) {
  constexpr int TILE = SC_THREADS * ITEMS;
  // the tile, padded so that thread-blocked and coalesced accesses are both
  // free of bank conflicts
  constexpr int PAD = 128 / sizeof(T);
  __shared__ T stage[TILE + TILE / PAD];
  auto at = [](int k) { return k + k / PAD; };
  const int tiles = (n + TILE - 1) / TILE;
  const bool resident = gridDim.x > 1 && tiles <= (int)gridDim.x;  // phase 1's loads kept
  T v[ITEMS];
  auto load = [&](int t) {
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const int i = t * TILE + r * SC_THREADS + threadIdx.x;
      v[r] = i < n ? f.value(i) : T(0);
    }
  };
  // 1. tile sums (fixed order), fallback state
  if (gridDim.x > 1) {
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      load(t);
      T s = T(0);
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) s += v[r];
      T total;
      sc_block_exclusive(s, &total);
      if (threadIdx.x == 0) tsum[t] = total;
#pragma unroll
      for (int r = 0; r < ITEMS; ++r) {
        const int i = t * TILE + r * SC_THREADS + threadIdx.x;
        if (i < n) f.fallback(i);
      }
    }
  }
  if (!grid_barrier(sync, fail)) {
    if (threadIdx.x == 0) f.failed();
    return;
  }
  // 2.-3. per tile: its prefix over the earlier tiles, then the items
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    T pre = T(0);
    if (gridDim.x > 1) {
      for (int c = 0; c * SC_THREADS < t; ++c) {  // tiles [0, t) in blocks of SC_THREADS
        const int j = c * SC_THREADS + threadIdx.x;
        T total;
        sc_block_exclusive(j < t ? __ldcg(&tsum[j]) : T(0), &total);
        pre += total;
      }
    }
    if (!resident) load(t);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) stage[at(r * SC_THREADS + threadIdx.x)] = v[r];
    __syncthreads();
    T b[ITEMS];
    T s = T(0);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      b[r] = stage[at(threadIdx.x * ITEMS + r)];
      s += b[r];
    }
    T total;
    T run = pre + sc_block_exclusive(s, &total);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      if (INCLUSIVE) {
        run += b[r];
        b[r] = run;
      } else {
        const T x = b[r];
        b[r] = run;
        run += x;
      }
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) stage[at(threadIdx.x * ITEMS + r)] = b[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const int i = t * TILE + r * SC_THREADS + threadIdx.x;
      if (i < n) f.emit(i, stage[at(r * SC_THREADS + threadIdx.x)], v[r]);
    }
    __syncthreads();  // stage reused
  }
  f.end();
}

// no-op hooks
struct ScanHooks {
  __device__ void fallback(int) const {}
  __device__ void failed() const {}
  __device__ void end() const {}
};

// out[i] = the sum (not overlapping in)
template <class T>
struct ScanArray : ScanHooks {
  const T *in;
  T *out;
  __device__ T value(int i) const { return in[i]; }
  __device__ void emit(int i, T pos, T) const { out[i] = pos; }
};

template <class T, bool INCLUSIVE, int ITEMS, class F>
void scan_launch(const F &f, int64_t n, int *fail, ZeroPool &zeroed, cudaStream_t s) {
  constexpr int TILE = SC_THREADS * ITEMS;
  const void *kern = (const void *)k_scan<T, INCLUSIVE, ITEMS, F>;
  const int64_t tiles = (n + TILE - 1) / TILE;
  const int g = tiles <= 1 ? 1 : (int)std::min<int64_t>(tiles, coop_blocks(kern, SC_THREADS, 0, 2));
  DevBuf<T> tsum;
  if (g > 1) tsum.alloc(tiles, s);
  int ni = (int)n;
  T *ts = tsum.get();
  RadixSync *sync = g > 1 ? zeroed.take<RadixSync>(1) : nullptr;
  void *args[] = {(void *)&f, (void *)&ni, (void *)&ts, (void *)&sync, (void *)&fail};
  launch_coop(kern, g, SC_THREADS, args, 0, s);
}

// emits item 0 + ... + item i - 1 (exclusive) or + item i (inclusive) for i < n;
// zeroed: where the barrier comes from.  Whole numbers may take the smaller
// tiles where these are no more than the SMs; floating point keeps one grouping.
template <class T, bool INCLUSIVE, class F>
void scan_each(const F &f, int64_t n, int *fail, ZeroPool &zeroed, cudaStream_t s) {
  if (n <= 0) return;
  FMMB_CHECK(n < (int64_t(1) << 30), ERR_INVALID_ARGUMENT, "scan: more than 2^30 elements");
  if constexpr (std::is_integral<T>::value)
    if (n > SC_THREADS * SC_ITEMS && n <= (int64_t)SC_THREADS * SC_FEW * 148) {
      scan_launch<T, INCLUSIVE, SC_FEW>(f, n, fail, zeroed, s);
      return;
    }
  scan_launch<T, INCLUSIVE, SC_ITEMS>(f, n, fail, zeroed, s);
}

// out[i] = in[0] + ... + in[i] (INCLUSIVE) or without in[i]; no overlap
template <class T, bool INCLUSIVE>
void prefix_sum(const T *in, T *out, int64_t n, int *fail, cudaStream_t s) {
  DevBuf<RadixSync> sync;
  sync.alloc(16, s);
  ZeroPool zeroed(sync.get(), 16 * sizeof(RadixSync), s);
  scan_each<T, INCLUSIVE>(ScanArray<T>{{}, in, out}, n, fail, zeroed, s);
}

}  // namespace
}  // namespace fmmb
