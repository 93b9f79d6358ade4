// Warp-level tensor-core GEMM helpers shared by the FMM passes.
#pragma once
#include "fmm.cuh"

namespace fmmb {

__host__ __device__ inline int pad_ld(int n) { return n + 4; }  // n multiple of 8 -> 4 or 12 mod 16

// D[8x8] += A[8x4] . B[4x8] on the FP64 tensor cores
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Warp tile: C[r0 + 8*rb + g][c0 + 8*cb*cstride + 2q + i] += sum_k A[.][k] * B[k][.]
// for rb < RB and the column blocks cb < CB that start below ncols
// (g = lane/4, q = lane%4; fragment layouts of mma.m8n8k4.f64).
// A: shared memory, row-major, stride lda.  B: shared memory, row-major [K][ldb].
template <int RB, int CB>
__device__ __forceinline__ void warp_gemm(const double *A, int lda, const double *B, int ldb, int K,
                                          int r0, int c0, int cstride, int ncols,
                                          double (&acc)[RB][CB][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const double *Ap = A + (r0 + g) * lda + q;
  const double *Bp = B + (size_t)q * ldb + c0 + g;
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    double a[RB], b[CB];
#pragma unroll
    for (int rb = 0; rb < RB; ++rb) a[rb] = Ap[8 * rb * lda + k];
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) {
      const double *bp = Bp + (size_t)k * ldb + 8 * cb * cstride;
      b[cb] = (c0 + 8 * cb * cstride < ncols) ? *bp : 0.0;
    }
#pragma unroll
    for (int rb = 0; rb < RB; ++rb)
#pragma unroll
      for (int cb = 0; cb < CB; ++cb)
        if (c0 + 8 * cb * cstride < ncols) dmma(acc[rb][cb], a[rb], b[cb]);
  }
}

// Asynchronous 16-byte global -> shared copy (cp.async, L2 only); complete
// after cp_async_wait_all() and, for other threads, a barrier.
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc) {
  const unsigned int d = static_cast<unsigned int>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Start copying a rows x cols row-major matrix (row stride cols) from global
// to shared memory with row stride ld; cols and ld are multiples of 16 bytes,
// both pointers 16-byte aligned.  Wait with cp_async_wait_all + barrier.
template <class T>
__device__ __forceinline__ void stage_rows(T *dst, int ld, const T *__restrict__ src, int rows,
                                           int cols) {
  constexpr int V = 16 / sizeof(T);
  const int cv = cols / V, n = rows * cv;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int r = i / cv, c = i - r * cv;
    cp_async16(dst + (size_t)r * ld + c * V, src + (size_t)i * V);
  }
}

// Shared-memory row stride (in floats) for a B operand of the split-TF32
// warp GEMMs: the four k-rows a warp reads start in distinct bank groups.
__host__ __device__ inline int ldb_f(int cols) { return (cols % 16 == 8) ? cols : cols + 8; }

template <int RB, int CB>
__device__ __forceinline__ void zero_acc(double (&acc)[RB][CB][2]) {
#pragma unroll
  for (int rb = 0; rb < RB; ++rb)
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) acc[rb][cb][0] = acc[rb][cb][1] = 0.0;
}

// Check-to-equivalent operators as a GEMM reads them: U and VH row-major
// with row stride ld, staged in shared memory.
struct C2EView {
  const double *u, *sinv, *vh;
  int ld;
};

// start staging a level's check-to-equivalent operators (U, 1/S, VH) in
// shared memory (asynchronous, see stage_rows): dst holds
// c2e_stage_doubles(np) doubles
__device__ __forceinline__ C2EView c2e_stage(const LevelOpsDev &op, int np, double *dst) {
  const int ld = pad_ld(np);
  double *u = dst, *vh = dst + np * ld, *si = dst + 2 * np * ld;
  stage_rows(u, ld, op.u, np, np);
  stage_rows(vh, ld, op.vh, np, np);
  stage_rows(si, np, op.sinv, 1, np);
  return {u, si, vh, ld};
}

__host__ __device__ inline int c2e_stage_doubles(int np) { return 2 * np * pad_ld(np) + np; }

// Check-to-equivalent on a 32-row tile: out = ((P . U) * sinv) . VH.
// P, T: shared [32][pad_ld(np)].  Row t goes to out_row[t] (np doubles) when
// out_row[t] is not null.  Starts and ends with a barrier-free read of P; the
// caller synchronises before.
__device__ inline void c2e_tile(const C2EView &op, int np, const double *P, double *T,
                                double *const *out_row) {
  const int ldp = pad_ld(np);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int r0 = 8 * (warp & 3), c0 = 8 * (warp >> 2);
  double acc[1][4][2];
  zero_acc(acc);
  warp_gemm<1, 4>(P, ldp, op.u, op.ld, np, r0, c0, 2, np, acc);
#pragma unroll
  for (int cb = 0; cb < 4; ++cb) {
    const int col = c0 + 16 * cb + 2 * q;
    if (col < np) {
      T[(r0 + g) * ldp + col] = acc[0][cb][0] * op.sinv[col];
      T[(r0 + g) * ldp + col + 1] = acc[0][cb][1] * op.sinv[col + 1];
    }
  }
  __syncthreads();
  zero_acc(acc);
  warp_gemm<1, 4>(T, ldp, op.vh, op.ld, np, r0, c0, 2, np, acc);
  double *o = out_row[r0 + g];
  if (o) {
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
      const int col = c0 + 16 * cb + 2 * q;
      if (col < np) *reinterpret_cast<double2 *>(o + col) = make_double2(acc[0][cb][0], acc[0][cb][1]);
    }
  }
}

__device__ __forceinline__ void cp_async_commit_group() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---- GEMMs with the operator in fragment order ----
// An operator B [K][N] (K, N multiples of 8) is stored as the mma.m8n8k4
// fragments its readers need: element (kp N/8 + cb) 32 + lane of an array of
// pairs holds B[8 kp + q][8 cb + g] and B[8 kp + 4 + q][8 cb + g] (g = lane/4,
// q = lane%4), so a warp reads two k-steps of a column block in one coalesced
// 512-byte load (from global memory) or without bank conflicts (from shared).
template <class F>
inline void pack_fragments(int K, int N, F &&at, double *dst) {
  for (int kp = 0; kp < K / 8; ++kp)
    for (int cb = 0; cb < N / 8; ++cb)
      for (int lane = 0; lane < 32; ++lane)
        for (int h = 0; h < 2; ++h)
          dst[((size_t(kp) * (N / 8) + cb) * 32 + lane) * 2 + h] =
              at(8 * kp + 4 * h + (lane & 3), 8 * cb + (lane >> 2));
}

// (volatile: the load stays where it is written, ahead of the DMMAs of the
// pairs before it; left to itself the compiler sinks it to its use)
__device__ __forceinline__ double2 load_pair(const double2 *p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

constexpr int FG_WARPS = 8;  // warps of a block that runs these tiles
constexpr int FG_PART = FG_WARPS * 64;  // doubles of the k-part exchange

// ---- tiles of 8 RB rows, the operator's fragments in shared memory ----
// The tile's units (row block, column block) are dealt out to the 8 warps, at
// most RB each; where there are no more than 4 of them the warps split the k
// range too (KS parts, summed through shared memory).
template <int RB>
struct UnitSplit {
  int ncb, n_units, u0, kpart, ks;
  __device__ explicit UnitSplit(int ncb_) : ncb(ncb_), n_units(RB * ncb_) {
    const int warp = threadIdx.x >> 5;
    ks = n_units <= FG_WARPS / 2 ? FG_WARPS / n_units : 1;
    u0 = ks > 1 ? warp % n_units : warp;
    kpart = ks > 1 ? warp / n_units : 0;
    if (kpart >= ks) u0 = n_units;  // no share
  }
  __device__ bool has(int i) const { return u0 + FG_WARPS * i < n_units && (i == 0 || ks == 1); }
  __device__ int rb(int i) const { return (u0 + FG_WARPS * i) / ncb; }
  __device__ int cb(int i) const { return (u0 + FG_WARPS * i) % ncb; }
};

// acc[i] += A[rows of unit i][8 k0 ..] . B; B's k pairs bstride column blocks
// apart.  A single unit alternates between two accumulators: one chain of
// dependent DMMAs (32 clocks each) would leave the pipe (18) half idle.
template <int RB>
__device__ __forceinline__ void unit_gemm(const UnitSplit<RB> &t, const double *A, int lda,
                                          const double2 *B, int bstride, int npairs,
                                          double (&acc)[RB][2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int k0 = npairs * t.kpart / t.ks, k1 = npairs * (t.kpart + 1) / t.ks;
  const double *Ap[RB];
  const double2 *Bp[RB];
#pragma unroll
  for (int i = 0; i < RB; ++i) {
    acc[i][0] = acc[i][1] = 0.0;
    const int j = t.has(i) ? i : 0;
    Ap[i] = A + (8 * t.rb(j) + g) * lda + q;
    Bp[i] = B + t.cb(j) * 32 + lane;
  }
  if (!t.has(0)) return;
  double odd[2] = {0.0, 0.0};
#pragma unroll 4
  for (int kp = k0; kp < k1; ++kp) {
#pragma unroll
    for (int i = 0; i < RB; ++i)
      if (i == 0 || t.has(i)) {
        const double2 b = Bp[i][kp * bstride * 32];
        const double a0 = Ap[i][8 * kp], a1 = Ap[i][8 * kp + 4];
        dmma(acc[i], a0, b.x);
        if (RB == 1)
          dmma(odd, a1, b.y);
        else
          dmma(acc[i], a1, b.y);
      }
  }
  if (RB == 1) {
    acc[0][0] += odd[0];
    acc[0][1] += odd[1];
  }
}

// sum the k parts into the warps of part 0 through part (FG_PART doubles); a
// barrier inside when there are several
template <int RB>
__device__ __forceinline__ void unit_sum(const UnitSplit<RB> &t, double (&acc)[RB][2], double *part) {
  if (t.ks == 1) return;
  const int lane = threadIdx.x & 31;
  if (t.has(0) && t.kpart > 0)
    *reinterpret_cast<double2 *>(part + (t.u0 * (t.ks - 1) + t.kpart - 1) * 64 + 2 * lane) =
        make_double2(acc[0][0], acc[0][1]);
  __syncthreads();
  if (t.has(0) && t.kpart == 0)
    for (int k = 0; k < t.ks - 1; ++k) {
      const double2 v =
          *reinterpret_cast<const double2 *>(part + (t.u0 * (t.ks - 1) + k) * 64 + 2 * lane);
      acc[0][0] += v.x;
      acc[0][1] += v.y;
    }
}

// f(row, column, accumulator pair) for the tile's summed results
template <int RB, class F>
__device__ __forceinline__ void unit_each(const UnitSplit<RB> &t, const double (&acc)[RB][2], F &&f) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  if (t.kpart == 0) {
#pragma unroll
    for (int i = 0; i < RB; ++i)
      if (t.has(i)) f(8 * t.rb(i) + g, 8 * t.cb(i) + 2 * q, acc[i][0], acc[i][1]);
  }
}

// Check-to-equivalent of a tile of 8 RB rows: ((P . U) diag(1/S)) . VH, P and T
// [8 RB][pad_ld(np)] and the operators in shared memory; row t goes to
// out_row[t] (np doubles) where that is not null.  The caller synchronises before.
template <int RB>
__device__ __forceinline__ void c2e_rows_smem(const double2 *U, const double2 *VH, const double *sinv,
                                              int np, const double *P, double *T, double *part,
                                              double *const *out_row) {
  const int ldp = pad_ld(np), ncb = np / 8;
  const UnitSplit<RB> t(ncb);
  double acc[RB][2];
  unit_gemm(t, P, ldp, U, ncb, ncb, acc);
  unit_sum(t, acc, part);
  unit_each(t, acc, [&](int r, int c, double a, double b) {
    *reinterpret_cast<double2 *>(T + r * ldp + c) = make_double2(a * sinv[c], b * sinv[c + 1]);
  });
  __syncthreads();
  unit_gemm(t, T, ldp, VH, ncb, ncb, acc);
  unit_sum(t, acc, part);
  unit_each(t, acc, [&](int r, int c, double a, double b) {
    double *o = out_row[r];
    if (o) *reinterpret_cast<double2 *>(o + c) = make_double2(a, b);
  });
}

// ---- bulk copies (one thread): global -> shared, counted by an mbarrier ----
__device__ __forceinline__ void bulk_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(bar))),
               "r"(bytes)
               : "memory");
}
// dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
      "l"(src), "r"(bytes), "r"(static_cast<uint32_t>(__cvta_generic_to_shared(bar)))
      : "memory");
}

}  // namespace fmmb
