// C-ABI entry points (include/flexmm_b200.h): operator sets, plans, passes.
#include <string.h>

#include <algorithm>
#include <cmath>

#include <map>
#include <atomic>
#include <cstddef>
#include <mutex>

#include <memory>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/flexmm_b200.h"
#include "fmm.cuh"
#include "gemm.cuh"
#include "timing.cuh"

using namespace fmmb;

namespace {
thread_local std::string g_last_error;

int fail(const Error &e) {
  g_last_error = e.what();
  return e.code;
}

template <class F>
int guarded(F &&f) {
  try {
    f();
    return FMM_OK;
  } catch (const Error &e) {
    return fail(e);
  } catch (const std::exception &e) {
    g_last_error = e.what();
    return FMM_ERR_INVALID_ARGUMENT;
  }
}

struct LevelEntry {
  DevBuf<double> buf;
  DevBuf<float> buf32;
  LevelOpsDev dev;
  DevBuf<LevelOpsDev> dev_copy;  // `dev` in device memory, gathered per plan by a kernel
  DevBuf<double> bb_m2l;  // black-box FMM: [40 np x np], the operators stacked, each transposed
  // black-box FMM: the common basis Q [np x 64] and its transpose [64 x np],
  // with the operators in it as M2L fragments (dev.m2l_f); or, at np <= 64, the
  // operators themselves as fragments (bb_fast without bb_q)
  DevBuf<double> bb_q, bb_frag;
  bool bb_fast = false;
  DevBuf<double> st;      // Stokes FMM: this width's operators (StokesArgs::Level layout)
  StokesArgs::Level st_lev{};
};

// round to TF32 (10 explicit mantissa bits), to nearest, ties away from zero
float tf32_rna(float x) {
  uint32_t u;
  memcpy(&u, &x, 4);
  if ((u & 0x7f800000u) != 0x7f800000u) u += 0x1000u;
  u &= 0xffffe000u;
  float r;
  memcpy(&r, &u, 4);
  return r;
}

int pad8(int n) { return (n + 7) & ~7; }

}  // namespace

void fmmb::smem_limit_impl(const void *kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, size_t> done;
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  size_t &have = done[{kernel, dev}];
  if (have >= bytes) return;
  FMMB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
  have = bytes;
}

size_t fmmb::smem_optin() {
  int dev = 0, v = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  FMMB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  return size_t(v);
}

int fmmb::coop_blocks(const void *kernel, int threads, size_t smem, int per_sm) {
  static std::mutex mu;
  static std::map<std::tuple<const void *, int, int, size_t>, std::pair<int, int>> known;
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  std::pair<int, int> &k = known[{kernel, dev, threads, smem}];  // SMs, blocks that fit on one
  if (k.first == 0) {
    int fit = 0, sms = 0;
    FMMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, smem));
    FMMB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    FMMB_CHECK(fit >= 1, ERR_CUDA, "cooperative kernel does not fit on an SM");
    k = {sms, fit};
  }
  return k.first * std::min(k.second, per_sm);
}

namespace {

// h_0 = e^x K0(x), h_1 = e^x K1(x) / x for x >= 1: trapezoidal rule on
// int_0^inf exp(-2x sinh^2(t/2)) cosh^n(t) dt (exponent without cancellation;
// step below the integrand's width 1/sqrt(x); summed from the small terms up)
long double bessel_h_host(int n, long double x) {
  const long double h = std::min(1.0L / 16.0L, 0.2L / std::sqrt(x));
  const int m = (int)std::ceil(std::acosh(1.0L + 60.0L / x) / h);
  long double s = 0.0L;
  for (int i = m; i >= 1; --i) {
    const long double t = i * h, sh = std::sinh(0.5L * t);
    s += std::exp(-2.0L * x * sh * sh) * (n ? std::cosh(t) : 1.0L);
  }
  s += 0.5L;  // t = 0
  return n ? h * s / x : h * s;
}

// the polynomials of h_0, h_1 on the eighths of the octaves (bessel.cuh):
// interpolation at Chebyshev nodes, rewritten in powers of x - c
const std::vector<double> &bessel_table_host() {
  static const std::vector<double> tab = [] {
    std::vector<double> t(BESSEL_TABLE_DOUBLES, 0.0);
    constexpr int N = BESSEL_NCOEF;
    const long double pi = std::acos(-1.0L);
    for (int n = 0; n < 2; ++n)
      for (int iv = 0; iv < BESSEL_INTERVALS; ++iv) {
        const long double a = std::ldexp(1.0L, iv / BESSEL_PARTS), hw = a / (2 * BESSEL_PARTS);
        const long double c = a + hw * (2 * (iv % BESSEL_PARTS) + 1);
        long double f[N], cheb[N];
        for (int k = 0; k < N; ++k) f[k] = bessel_h_host(n, c + hw * std::cos(pi * (k + 0.5L) / N));
        for (int i = 0; i < N; ++i) {
          long double v = 0.0L;
          for (int k = 0; k < N; ++k) v += f[k] * std::cos(pi * i * (k + 0.5L) / N);
          cheb[i] = (i == 0 ? 1.0L : 2.0L) * v / N;
        }
        // sum_i cheb_i T_i(u), T_i in powers of u = (x - c) / hw
        long double pow[N] = {}, t0[N] = {1.0L}, t1[N] = {0.0L, 1.0L};
        for (int i = 0; i < N; ++i) {
          for (int k = 0; k < N; ++k) pow[k] += cheb[i] * t0[k];
          long double t2[N];
          for (int k = 0; k < N; ++k) t2[k] = (k ? 2.0L * t1[k - 1] : 0.0L) - t0[k];
          std::copy(t1, t1 + N, t0);
          std::copy(t2, t2 + N, t1);
        }
        long double scale = 1.0L;
        for (int k = 0; k < N; ++k, scale /= hw)
          t[(n * BESSEL_INTERVALS + iv) * BESSEL_ROW + k] = double(pow[k] * scale);
      }
    return t;
  }();
  return tab;
}

// the Bessel tables on the current device (uploaded once per device, kept
// until exit)
const double *bessel_table_device() {
  static std::mutex mu;
  static std::map<int, double *> per_device;
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  auto it = per_device.find(dev);
  if (it != per_device.end()) return it->second;
  const std::vector<double> &h = bessel_table_host();
  double *d = nullptr;
  FMMB_CUDA(cudaMalloc((void **)&d, h.size() * sizeof(double)));
  FMMB_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
  per_device[dev] = d;
  return d;
}

// tabulated radial kernels registered by fmm_kernel_table_create: host
// coefficients plus their per-device copies (kept until exit)
struct RadialTable {
  int j0, noct, ncheb;
  std::vector<double> coef;
  std::map<int, double *> dev;
};
std::mutex g_tables_mu;
std::vector<std::unique_ptr<RadialTable>> g_tables;

bool kernel_known(int kernel_id) {
  return kernel_id == KERNEL_LAPLACE || kernel_id == KERNEL_MOD_HELMHOLTZ ||
         kernel_id == KERNEL_RADIAL_TABLE;
}

// a kernel's device parameters: the caller's values plus the tables it reads
KernelParams kernel_params(int kernel_id, const double *kparams) {
  KernelParams kp{};
  for (int i = 0; i < 4; ++i) kp.p[i] = kparams ? kparams[i] : 0.0;
  kp.table = nullptr;
  if (kernel_id == KERNEL_MOD_HELMHOLTZ) {
    FMMB_CHECK(kp.p[0] > 0.0, ERR_INVALID_ARGUMENT, "modified Helmholtz needs k = kparams[0] > 0");
    kp.table = bessel_table_device();
  }
  if (kernel_id == KERNEL_RADIAL_TABLE) {
    std::lock_guard<std::mutex> g(g_tables_mu);
    const int id = int(kp.p[0]);
    FMMB_CHECK(kp.p[0] == double(id) && id >= 0 && id < (int)g_tables.size() && g_tables[id],
               ERR_INVALID_ARGUMENT, "kparams[0] is not a table id from fmm_kernel_table_create");
    RadialTable &t = *g_tables[id];
    int dev = 0;
    FMMB_CUDA(cudaGetDevice(&dev));
    if (!t.dev.count(dev)) {
      // rows of coefficient pairs: an odd count is filled up with a zero
      const int row = (t.ncheb + 1) / 2 * 2;
      std::vector<double> h((size_t)t.noct * row, 0.0);
      for (int o = 0; o < t.noct; ++o)
        std::copy_n(t.coef.data() + (size_t)o * t.ncheb, t.ncheb, h.data() + (size_t)o * row);
      double *d = nullptr;
      FMMB_CUDA(cudaMalloc((void **)&d, h.size() * sizeof(double)));
      FMMB_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
      t.dev[dev] = d;
    }
    kp.table = t.dev[dev];
    kp.p[1] = t.j0;
    kp.p[2] = t.noct;
    kp.p[3] = t.ncheb;
  }
  return kp;
}

bool kernel_scaled(int kernel_id) {
  switch (kernel_id) {
    case KERNEL_LAPLACE: return LaplaceF32::kScaled;
    default: return false;
  }
}

// kernels with an FP32 form for the mixed passes
bool kernel_mixed(int kernel_id) {
  return kernel_id == KERNEL_LAPLACE || kernel_id == KERNEL_MOD_HELMHOLTZ;
}

double kernel_offset(int kernel_id, const KernelParams &kp, double w) {
  switch (kernel_id) {
    case KERNEL_LAPLACE: return LaplaceF32::offset(w, kp);
    default: return 0.0;
  }
}

// Keep freed stream-ordered allocations in this process's default pool, so
// that plans created repeatedly reuse device memory instead of returning it
// to the driver at every synchronisation.
void retain_pool_memory() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  static thread_local int done_for = -1;
  if (done_for == dev) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    uint64_t keep = ~uint64_t(0);
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    // headroom reserved once: plans built while earlier ones are still
    // queued (a host running steps ahead) then take memory the pool already
    // maps, instead of mapping more in the middle of a step (milliseconds)
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) {
      const size_t want = std::min<size_t>(size_t(1) << 30, free_b / 8);
      void *p = nullptr;
      if (want > 0 && cudaMallocAsync(&p, want, 0) == cudaSuccess) {
        cudaFreeAsync(p, 0);
        cudaStreamSynchronize(0);
      }
    }
  }
  done_for = dev;
}

// The black-box M2M operator [p^2 x 4 p^2] as tensor factors: child c's block is
// X_c (x) Y_c, read off its first rows and columns (T_0 = 1 keeps its value under
// a shift, so X_c[0][0] = Y_c[0][0] = 1).  False where that is not the operator to
// 6e-15 of its largest element (the factors of the Chebyshev shift reproduce it
// to 5e-15 at most, p = 2 .. 16; any other is applied as it is).  Fragments for k_bb_shift
// (bbfmm.cu): M2M's Y and X, then L2L's, Y^T and X^T, each [4][P x P], P = 8 or 16.
bool bb_shift_fragments(int p, const double *m2mc, std::vector<double> &out) {
  const int n = p * p, P = p <= 8 ? 8 : 16;
  auto at = [&](int c, int a, int b, int a1, int b1) {
    return m2mc[size_t(a * p + b) * 4 * n + c * n + a1 * p + b1];
  };
  auto X = [&](int c, int a, int a1) { return a < p && a1 < p ? at(c, a, 0, a1, 0) : 0.0; };
  auto Y = [&](int c, int b, int b1) { return b < p && b1 < p ? at(c, 0, b, 0, b1) : 0.0; };
  double big = 0.0, off = 0.0;
  for (int c = 0; c < 4; ++c)
    for (int a = 0; a < p; ++a)
      for (int b = 0; b < p; ++b)
        for (int a1 = 0; a1 < p; ++a1)
          for (int b1 = 0; b1 < p; ++b1) {
            const double v = at(c, a, b, a1, b1);
            big = std::max(big, std::fabs(v));
            const double d = std::fabs(v - X(c, a, a1) * Y(c, b, b1));
            if (!(d <= off)) off = d;  // (NaN stays)
          }
  if (!(off <= 6e-15 * big)) return false;
  const size_t F = size_t(4) * P * P;
  out.assign(4 * F, 0.0);
  const int NB = P / 8, KS = P / 4;
  for (int t = 0; t < 2; ++t)  // M2M, L2L
    for (int c = 0; c < 4; ++c)
      for (int i = 0; i < NB; ++i)
        for (int lane = 0; lane < 32; ++lane) {
          const int g = lane >> 2, q = lane & 3;
          for (int ks = 0; ks < KS; ++ks) {
            const int r = 8 * i + g, k = 4 * ks + q;
            out[2 * t * F + ((size_t(c) * NB + i) * KS + ks) * 32 + lane] = t ? Y(c, k, r) : Y(c, r, k);
          }
          for (int cb = 0; cb < NB; ++cb)
            for (int h = 0; h < 2; ++h) {
              const int r = 8 * i + g, k = 8 * cb + 2 * q + h;
              out[(2 * t + 1) * F + (((size_t(c) * NB + i) * NB + cb) * 2 + h) * 32 + lane] =
                  t ? X(c, k, r) : X(c, r, k);
            }
        }
  return true;
}

// the 40 M2L operators of a black-box width as fragments: at(o, k, i) = column
// k (source), row i (target) of offset o's operator; present[o] = 0: none
template <class F>
void bb_fragments(LevelEntry &e, int np, const int *present, F &&at) {
  const size_t sq = size_t(np) * np;
  std::vector<double> f(sq * N_OFFSETS, 0.0);
  for (int o = 0; o < N_OFFSETS; ++o)
    if (present[o]) pack_fragments(np, np, [&](int k, int i) { return at(o, k, i); }, f.data() + o * sq);
  e.bb_frag.alloc(f.size(), 0);
  FMMB_CUDA(cudaMemcpy(e.bb_frag.get(), f.data(), f.size() * sizeof(double), cudaMemcpyHostToDevice));
  for (int o = 0; o < N_OFFSETS; ++o) {
    e.dev.kind[o] = present[o] ? M2L_DENSE : M2L_NULL;
    e.dev.m2l_f[o] =
        present[o] ? reinterpret_cast<const double2 *>(e.bb_frag.get() + o * sq) : nullptr;
  }
  e.bb_fast = true;
}
}  // namespace

constexpr int METHOD_KIFMM = 0, METHOD_BBFMM = 1, METHOD_STOKES = 2;

struct fmm_ops {
  int kernel_id;
  KernelParams kp;
  int neq, np;
  int method = METHOD_KIFMM;
  int p = 0;                  // black-box FMM: Chebyshev order
  DevBuf<double> bb_m2mc;     // black-box FMM: M2MC [np x 4np]
  DevBuf<double> bb_m2mct;    // and its transpose [4np x np]
  DevBuf<double> bb_sep;      // tensor factors of both (bb_shift_fragments); empty: none
  // what the plans of this set did last (fmm_plan::split_expected): a new plan's guess
  std::atomic<bool> split_expected{true};
  std::vector<std::unique_ptr<LevelEntry>> levels;
};

struct fmm_plan {
  fmm_ops *ops;
  cudaStream_t stream;
  TreeDev td;
  TreeHost th;
  std::vector<int> bound;  // per level: ops entry id or -1
  DevBuf<LevelOpsDev> ops_dev;
  DevBuf<double> tau_s, mult, ple, loc;
  DevBuf<float> mult32, loc32;  // mixed precision: FP32 expansions ...
  DevBuf<float> mult_tc;        // ... multipoles split TF32 hi / lo ...
  DevBuf<double> msum, lsum;    // ... and their FP64 component sums
  DevBuf<double> tsum;          // per node: FP64 sum of its charges
  // FP64 level passes: their barriers (upward, downward) and, as the third's
  // timeout, their failure flag; zeroed by each build
  DevBuf<RadixSync> sync;
  int *pass_fail() const { return sync.get() ? &sync.get()[2].timeout : nullptr; }
  DevBuf<int> err;              // set by kernels whose bounded waits ran out
  int precision = PREC_FP64;
  bool moved = false;  // sources moved on the frozen tree: a box no longer bounds its own
  bool have_expansions = false;
  DevBuf<double> tau2_s, partial;  // Stokes FMM: sorted fy; partial multipoles
  int n_rhs = 1;                   // charge columns of the last build (multi-RHS)
  // split own-source evaluation (near field on a side stream, see SplitEval):
  // `ready` is recorded once a single-column KIFMM build has sorted its charges
  DevBuf<double> dvx, dvy;  // dipole sources: strength * normal, sorted (see PassArgs)
  bool has_dipoles = false;
  DevBuf<double> st_dip;    // Stokes stresslets: sigma_x, sigma_y, n_x, n_y, sorted ([4][n])
  bool has_st_dipoles = false;
  cudaStream_t side = nullptr;  // from the device's pool, not owned
  cudaStream_t pass = nullptr;  // the pair's high-priority stream (PassStream)
  // Whether the expansions will be evaluated split, so that the build takes the
  // scratch and the high-priority stream for it: as the last ones were (the
  // first build: as the last of the operator set's were; -1 before it).  A guess
  // for speed alone: a split evaluation without either gives the same bits.
  int split_expected = -1;
  bool split_since_build = false;
  bool split_scratch_ready = false;  // allocated for this tree, before its ev_ready
  cudaEvent_t ev_ready = nullptr, ev_near = nullptr, ev_far = nullptr, ev_pass = nullptr;
  bool ready_recorded = false;
  // mixed form: the split near field pauses during the M2L (SplitEval::hold)
  cudaEvent_t ev_m2l = nullptr;
  DevBuf<int> near_hold;
  SplitScratch split_scratch;  // see split_scratch_prepare
  bool hold_armed = false;
  ~fmm_plan() {
    for (cudaEvent_t e : {ev_ready, ev_near, ev_far, ev_m2l, ev_pass})
      if (e) cudaEventDestroy(e);
  }
};

namespace {
// Streams beside the caller's: a few pairs of non-blocking streams per device,
// handed to plans round-robin (created once, kept until exit).  g_side runs
// the split evaluation's near field at the lowest priority, g_pass the FP64
// level passes at the highest: wherever a near-field block ends, a waiting
// block of a level pass goes first, so the chain of levels is not held up by
// the work it runs beside.
constexpr int SIDE_STREAMS = 8;
constexpr int SIDE_MAX_DEVICES = 64;
std::mutex g_side_mu;
cudaStream_t g_side[SIDE_MAX_DEVICES][SIDE_STREAMS] = {};
cudaStream_t g_pass[SIDE_MAX_DEVICES][SIDE_STREAMS] = {};
int g_side_next[SIDE_MAX_DEVICES] = {};

cudaStream_t side_stream(cudaStream_t *pass) {
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  FMMB_CHECK(dev >= 0 && dev < SIDE_MAX_DEVICES, ERR_UNSUPPORTED, "device ordinal too large");
  std::lock_guard<std::mutex> g(g_side_mu);
  if (!g_side[dev][0])  // all at once: no plan after the first pays for a stream
  {
    int least = 0, greatest = 0;
    FMMB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    for (int k = 0; k < SIDE_STREAMS; ++k) {
      FMMB_CUDA(cudaStreamCreateWithPriority(&g_pass[dev][k], cudaStreamNonBlocking, greatest));
      FMMB_CUDA(cudaStreamCreateWithPriority(&g_side[dev][k], cudaStreamNonBlocking, least));
    }
  }
  const int k = g_side_next[dev]++ % SIDE_STREAMS;
  *pass = g_pass[dev][k];
  return g_side[dev][k];
}

// Whether own-source evaluation runs split (near field beside the level
// passes).  Measured, off and on: a step of 1M clustered sources 2.35 and 2.28
// ms, of 200k with K0 0.96 and 0.85, a product on 250k ring points 0.56 and 0.50;
// the mixed form, whose near field pauses while the persistent tcgen05 M2L
// runs, 1.21 and 1.18 ms at 1M.  On for both by default;
// FLEXMM_B200_SPLIT_EVAL=0 turns it off, =1 on.
std::atomic<int> g_split_mode{-2};  // -2: not yet read from the environment

bool split_enabled(int precision) {
  int mode = g_split_mode.load(std::memory_order_relaxed);
  if (mode == -2) {
    const char *e = getenv("FLEXMM_B200_SPLIT_EVAL");
    int env = e ? (e[0] == '0' ? 0 : 1) : -1;
    g_split_mode.compare_exchange_strong(mode, env);
    mode = g_split_mode.load(std::memory_order_relaxed);
  }
  (void)precision;  // the same default for both forms
  return mode < 0 || mode == 1;
}

// the plan's split-evaluation events (created on first use) and side stream
void split_prepare(fmm_plan *p) {
  if (!p->side) p->side = side_stream(&p->pass);
  for (cudaEvent_t *e : {&p->ev_ready, &p->ev_near, &p->ev_far, &p->ev_m2l, &p->ev_pass})
    if (!*e) FMMB_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return st != cudaStreamCaptureStatusNone;
}

// The scratch of the split evaluation that is expected, ahead of ev_ready; given
// back where none is.  (Plans that evaluate gradients or other points only held
// it for nothing: the first pass of a new batch of 12 Stokes problems, whose
// adjoint evaluates Laplace gradients, 15.4 -> 13.9 ms.)
void split_scratch_prepare(fmm_plan *p, cudaStream_t s) {
  p->split_since_build = p->split_scratch_ready = false;
  if (p->split_expected < 0) p->split_expected = p->ops->split_expected;
  if (capturing(s)) return;
  if (!p->split_expected || !split_enabled(p->precision)) {
    p->split_scratch.release();
  } else {
    p->split_scratch.alloc(p->th.n_total(), p->th.n_points, p->precision == PREC_MIXED, s);
    p->split_scratch_ready = true;
  }
}

// what an evaluation of a plan's expansions says about the next ones
void split_note(fmm_plan *p, bool split) {
  if (p->split_since_build) return;
  p->split_since_build = split;
  p->split_expected = split;
  p->ops->split_expected = split;
}

// The stream of a plan's FP64 level passes: the high-priority one of its pair,
// which waits for ev_ready and which the caller's stream waits for at join()
// (at the latest when this object ends, so that buffers freed in the caller's
// stream order are no longer read).  The passes stay on the caller's stream
// where no near field is expected beside them (a plan that evaluates gradients
// or other points only: a batch of 12 on 8 streams of its own takes 7.9 ms that
// way, 8.8 ms through the pairs), and where that stream is being captured (the
// pool's streams are shared with plans outside the capture).
class PassStream {
 public:
  PassStream(fmm_plan *p, cudaStream_t s) : p_(p), s_(s), ps_(s) {
    const bool near_beside = split_enabled(PREC_FP64) && p->split_expected;
    if (!near_beside || capturing(s)) return;
    FMMB_CUDA(cudaStreamWaitEvent(p->pass, p->ev_ready, 0));
    ps_ = p->pass;
  }
  PassStream(const PassStream &) = delete;
  PassStream &operator=(const PassStream &) = delete;
  ~PassStream() {
    if (ps_ != s_ && cudaEventRecord(p_->ev_pass, ps_) == cudaSuccess)
      cudaStreamWaitEvent(s_, p_->ev_pass, 0);
  }
  cudaStream_t stream() const { return ps_; }
  void join() {
    if (ps_ == s_) return;
    FMMB_CUDA(cudaEventRecord(p_->ev_pass, ps_));
    ps_ = s_;
    FMMB_CUDA(cudaStreamWaitEvent(s_, p_->ev_pass, 0));
  }

 private:
  fmm_plan *p_;
  cudaStream_t s_, ps_;
};

// Zeroes up to 8 device buffers in one launch (instead of one memset each:
// at the start of build_expansions these sit between the tree and the first
// pass, where every launch's host and GPU overhead is on the critical path)
struct ZeroList {
  unsigned char *p[8];
  size_t bytes[8];
  int n;
};

__global__ void k_zero_buffers(ZeroList z) {
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t nthr = (size_t)gridDim.x * blockDim.x;
  for (int b = 0; b < z.n; ++b) {
    const size_t n16 = z.bytes[b] / 16;  // buffers are 16-byte aligned (checked by the host)
    uint4 *w = reinterpret_cast<uint4 *>(z.p[b]);
    for (size_t i = tid; i < n16; i += nthr) w[i] = make_uint4(0u, 0u, 0u, 0u);
    for (size_t i = 16 * n16 + tid; i < z.bytes[b]; i += nthr) z.p[b][i] = 0;
  }
}

class ZeroBatch {
 public:
  explicit ZeroBatch(cudaStream_t s) : s_(s) {}
  template <class T>
  ZeroBatch &add(DevBuf<T> &b) {
    if (!b.n) return *this;
    if (z_.n == 8 || (reinterpret_cast<uintptr_t>(b.get()) & 15)) {
      b.zero(s_);
      return *this;
    }
    z_.p[z_.n] = reinterpret_cast<unsigned char *>(b.get());
    z_.bytes[z_.n++] = b.n * sizeof(T);
    return *this;
  }
  void run() {
    if (!z_.n) return;
    size_t total = 0;
    for (int i = 0; i < z_.n; ++i) total += z_.bytes[i];
    int dev = 0, sms = 0;
    FMMB_CUDA(cudaGetDevice(&dev));
    FMMB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = (int)std::min<size_t>(size_t(sms) * 8, std::max<size_t>(1, total / 4096));
    k_zero_buffers<<<blocks, 256, 0, s_>>>(z_);
    FMMB_CUDA(cudaGetLastError());
    z_.n = 0;
  }

 private:
  cudaStream_t s_;
  ZeroList z_{};
};
}  // namespace

extern "C" {

const char *fmm_last_error(void) { return g_last_error.c_str(); }

int fmm_ops_create(int kernel_id, const double *kparams, int nequiv, fmm_ops **out) {
  return guarded([&] {
    FMMB_CHECK(out, ERR_INVALID_ARGUMENT, "out is NULL");
    FMMB_CHECK(kernel_known(kernel_id), ERR_UNSUPPORTED, "unknown kernel id");
    FMMB_CHECK(nequiv >= 1 && nequiv <= FMM_MAX_NEQUIV, ERR_INVALID_ARGUMENT,
               "nequiv must be in [1, 64]");
    const KernelParams kp = kernel_params(kernel_id, kparams);
    auto *o = new fmm_ops();
    o->kernel_id = kernel_id;
    o->kp = kp;
    o->neq = nequiv;
    o->np = pad8(nequiv);
    *out = o;
  });
}

int fmm_ops_add(fmm_ops *ops, const fmm_level_ops *lv, int *level_id) {
  return guarded([&] {
    FMMB_CHECK(ops && lv && level_id, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(ops->method == METHOD_KIFMM, ERR_INVALID_ARGUMENT,
               "black-box and Stokes operator sets take fmm_bb_ops_add / fmm_stokes_ops_add");
    const int n = ops->neq, np = ops->np;
    // host staging in the padded device layout
    std::vector<double> h;
    auto take = [&](size_t count) {
      size_t at = h.size();
      h.resize(at + ((count + 1) & ~size_t(1)), 0.0);  // keep 16-byte alignment
      return at;
    };
    const size_t o_lx = take(np), o_ly = take(np), o_u = take(size_t(np) * np), o_s = take(np),
                 o_vh = take(size_t(np) * np), o_uf = take(size_t(np) * np),
                 o_vhf = take(size_t(np) * np), o_m2mf = take(size_t(4) * np * np),
                 o_l2lf = take(size_t(4) * np * np);
    for (int k = 0; k < n; ++k) {
      h[o_lx + k] = lv->large_x[k];
      h[o_ly + k] = lv->large_y[k];
      h[o_s + k] = lv->c2e_sinv[k];
    }
    for (int i = 0; i < n; ++i)
      for (int k = 0; k < n; ++k) {
        h[o_u + size_t(i) * np + k] = lv->c2e_u[size_t(i) * n + k];
        h[o_vh + size_t(i) * np + k] = lv->c2e_vh[size_t(i) * n + k];
      }
    auto u_at = [&](int i, int k) { return h[o_u + size_t(i) * np + k]; };
    auto vh_at = [&](int i, int k) { return h[o_vh + size_t(i) * np + k]; };
    // M2MC[i][c Neq + k] at (row i, child c, k), 0 in the padding
    auto m2mc_at = [&](int i, int ck) {
      const int c = ck / np, k = ck % np;
      return i < n && k < n ? lv->m2mc[size_t(i) * 4 * n + c * n + k] : 0.0;
    };
    pack_fragments(np, np, u_at, h.data() + o_uf);
    pack_fragments(np, np, vh_at, h.data() + o_vhf);
    pack_fragments(4 * np, np, [&](int ck, int i) { return m2mc_at(i, ck); }, h.data() + o_m2mf);
    pack_fragments(np, 4 * np, m2mc_at, h.data() + o_l2lf);
    size_t o_m2l[FMM_N_OFFSETS];
    // mixed precision: dense operators minus their mean, as TF32 hi + lo
    std::vector<float> f;
    auto takef = [&](size_t count) {
      size_t at = f.size();
      f.resize(at + ((count + 3) & ~size_t(3)), 0.f);  // 16-byte aligned blocks
      return at;
    };
    auto split = [&](double v, size_t hi_at, size_t lo_at) {
      const float hi = tf32_rna((float)v);
      f[hi_at] = hi;
      f[lo_at] = tf32_rna((float)(v - (double)hi));
    };
    // FP32 evaluations of scale-invariant kernels work in width units
    const bool scaled = kernel_scaled(ops->kernel_id);
    FMMB_CHECK(!scaled || lv->width > 0, ERR_INVALID_ARGUMENT, "level width must be positive");
    const double inv_w = scaled ? 1.0 / lv->width : 1.0;
    const size_t f_lx = takef(np), f_ly = takef(np);
    float reach = 0.f;
    for (int k = 0; k < n; ++k) {
      f[f_lx + k] = (float)(lv->large_x[k] * inv_w);
      f[f_ly + k] = (float)(lv->large_y[k] * inv_w);
      reach = std::max({reach, std::fabs(f[f_lx + k]), std::fabs(f[f_ly + k])});
    }
    double c_m2m = 0.0;
    for (size_t i = 0; i < size_t(n) * 4 * n; ++i) c_m2m += lv->m2mc[i];
    c_m2m /= double(n) * 4 * n;
    const size_t f_m2mct_h = takef(size_t(4) * np * np), f_m2mct_l = takef(size_t(4) * np * np);
    const size_t f_m2mc_h = takef(size_t(4) * np * np), f_m2mc_l = takef(size_t(4) * np * np);
    for (int i = 0; i < n; ++i)
      for (int c = 0; c < 4; ++c)
        for (int k = 0; k < n; ++k) {
          const double v = lv->m2mc[size_t(i) * 4 * n + c * n + k] - c_m2m;
          const size_t t1 = size_t(c * np + k) * np + i, t2 = size_t(i) * 4 * np + c * np + k;
          split(v, f_m2mct_h + t1, f_m2mct_l + t1);
          split(v, f_m2mc_h + t2, f_m2mc_l + t2);
        }
    size_t f_m2l_h[FMM_N_OFFSETS], f_m2l_l[FMM_N_OFFSETS];
    size_t f_tc_h[FMM_N_OFFSETS], f_tc_l[FMM_N_OFFSETS];
    const int ntc = (np + 15) & ~15;  // tensor-core N: multiple of 16
    double c_m2l[FMM_N_OFFSETS];
    std::vector<double> dense(size_t(n) * n);
    for (int o = 0; o < FMM_N_OFFSETS; ++o) {
      const int r = lv->m2l_rank[o];
      c_m2l[o] = 0.0;
      o_m2l[o] = 0;
      f_m2l_h[o] = f_m2l_l[o] = f_tc_h[o] = f_tc_l[o] = 0;
      if (r == 0) continue;
      if (r < 0) {
        for (size_t i = 0; i < size_t(n) * n; ++i) dense[i] = lv->m2l_a[o][i];
      } else {  // the truncated operator M2 . M1, as the reference applies it
        FMMB_CHECK(r <= n, ERR_INVALID_ARGUMENT, "M2L rank exceeds nequiv");
        for (int i = 0; i < n; ++i)
          for (int k = 0; k < n; ++k) {
            double acc = 0.0;
            for (int q = 0; q < r; ++q) acc += lv->m2l_a[o][size_t(i) * r + q] * lv->m2l_b[o][size_t(q) * n + k];
            dense[size_t(i) * n + k] = acc;
          }
      }
      o_m2l[o] = take(size_t(np) * np);  // D^T: row k (source), column i (target)
      pack_fragments(np, np, [&](int k, int i) {
        return i < n && k < n ? dense[size_t(i) * n + k] : 0.0;
      }, h.data() + o_m2l[o]);
      double c = 0.0;
      for (size_t i = 0; i < size_t(n) * n; ++i) c += dense[i];
      c /= double(n) * n;
      c_m2l[o] = c;
      f_m2l_h[o] = takef(size_t(np) * np);
      f_m2l_l[o] = takef(size_t(np) * np);
      f_tc_h[o] = takef(size_t(ntc) * np);
      f_tc_l[o] = takef(size_t(ntc) * np);
      for (int i = 0; i < n; ++i)
        for (int k = 0; k < n; ++k) {
          const size_t t = size_t(k) * np + i;  // B layout [K = source comp][N = target comp]
          split(dense[size_t(i) * n + k] - c, f_m2l_h[o] + t, f_m2l_l[o] + t);
          const size_t u = size_t(i) * np + k;  // tcgen05 B: N x K, K-major
          split(dense[size_t(i) * n + k] - c, f_tc_h[o] + u, f_tc_l[o] + u);
        }
    }
    auto e = std::make_unique<LevelEntry>();
    e->buf32.alloc(f.size(), 0);
    FMMB_CUDA(cudaMemcpy(e->buf32.get(), f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice));
    {
      float *fb = e->buf32.get();
      e->dev.lx32 = fb + f_lx;
      e->dev.ly32 = fb + f_ly;
      e->dev.m2mct_hi = fb + f_m2mct_h;
      e->dev.m2mct_lo = fb + f_m2mct_l;
      e->dev.m2mc_hi = fb + f_m2mc_h;
      e->dev.m2mc_lo = fb + f_m2mc_l;
      e->dev.c_m2m = c_m2m;
      e->dev.inv_w = inv_w;
    e->dev.reach32 = reach;
      e->dev.kofs = scaled ? kernel_offset(ops->kernel_id, ops->kp, lv->width) : 0.0;
      for (int o = 0; o < FMM_N_OFFSETS; ++o) {
        e->dev.m2l_hi[o] = lv->m2l_rank[o] == 0 ? nullptr : fb + f_m2l_h[o];
        e->dev.m2l_lo[o] = lv->m2l_rank[o] == 0 ? nullptr : fb + f_m2l_l[o];
        e->dev.m2l_tc_hi[o] = lv->m2l_rank[o] == 0 ? nullptr : fb + f_tc_h[o];
        e->dev.m2l_tc_lo[o] = lv->m2l_rank[o] == 0 ? nullptr : fb + f_tc_l[o];
        e->dev.c_m2l[o] = c_m2l[o];
      }
    }
    e->buf.alloc(h.size(), 0);
    FMMB_CUDA(cudaMemcpy(e->buf.get(), h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    double *b = e->buf.get();
    e->dev.lx = b + o_lx;
    e->dev.ly = b + o_ly;
    e->dev.u = b + o_u;
    e->dev.sinv = b + o_s;
    e->dev.vh = b + o_vh;
    e->dev.u_f = reinterpret_cast<const double2 *>(b + o_uf);
    e->dev.vh_f = reinterpret_cast<const double2 *>(b + o_vhf);
    e->dev.m2m_f = reinterpret_cast<const double2 *>(b + o_m2mf);
    e->dev.l2l_f = reinterpret_cast<const double2 *>(b + o_l2lf);
    for (int o = 0; o < FMM_N_OFFSETS; ++o) {
      const bool null = lv->m2l_rank[o] == 0;
      e->dev.m2l_f[o] = null ? nullptr : reinterpret_cast<const double2 *>(b + o_m2l[o]);
      e->dev.kind[o] = null ? M2L_NULL : M2L_DENSE;
    }
    e->dev_copy.alloc(1, 0);
    FMMB_CUDA(cudaMemcpy(e->dev_copy.get(), &e->dev, sizeof(LevelOpsDev), cudaMemcpyHostToDevice));
    ops->levels.push_back(std::move(e));
    *level_id = int(ops->levels.size()) - 1;
  });
}

int fmm_bb_ops_create(int kernel_id, const double *kparams, int p, const double *m2mc,
                      fmm_ops **out) {
  return guarded([&] {
    FMMB_CHECK(out && m2mc, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(kernel_known(kernel_id), ERR_UNSUPPORTED, "unknown kernel id");
    FMMB_CHECK(p >= 2 && p <= FMM_BB_MAX_P, ERR_INVALID_ARGUMENT, "p must be in [2, 16]");
    const KernelParams kp = kernel_params(kernel_id, kparams);
    const int n = p * p, np = pad8(n);
    std::vector<double> h(size_t(np) * 4 * np, 0.0);
    for (int i = 0; i < n; ++i)
      for (int c = 0; c < 4; ++c)
        for (int k = 0; k < n; ++k) h[size_t(i) * 4 * np + c * np + k] = m2mc[size_t(i) * 4 * n + c * n + k];
    auto o = std::make_unique<fmm_ops>();
    o->kernel_id = kernel_id;
    o->kp = kp;
    o->neq = n;
    o->np = np;
    o->method = METHOD_BBFMM;
    o->p = p;
    o->bb_m2mc.alloc(h.size(), 0);
    FMMB_CUDA(cudaMemcpy(o->bb_m2mc.get(), h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    std::vector<double> ht(h.size(), 0.0);  // [4np x np]: the M2M row GEMM's operator
    for (int i = 0; i < np; ++i)
      for (int k = 0; k < 4 * np; ++k) ht[size_t(k) * np + i] = h[size_t(i) * 4 * np + k];
    o->bb_m2mct.alloc(ht.size(), 0);
    FMMB_CUDA(cudaMemcpy(o->bb_m2mct.get(), ht.data(), ht.size() * sizeof(double),
                         cudaMemcpyHostToDevice));
    std::vector<double> sep;
    if (bb_shift_fragments(p, m2mc, sep)) {
      o->bb_sep.alloc(sep.size(), 0);
      FMMB_CUDA(cudaMemcpy(o->bb_sep.get(), sep.data(), sep.size() * sizeof(double),
                           cudaMemcpyHostToDevice));
    }
    *out = o.release();
  });
}

int fmm_bb_ops_add(fmm_ops *ops, const fmm_bb_level_ops *lv, int *level_id) {
  return guarded([&] {
    FMMB_CHECK(ops && lv && level_id && lv->m2l_rank, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(ops->method == METHOD_BBFMM, ERR_INVALID_ARGUMENT,
               "fmm_bb_ops_add needs a black-box operator set (fmm_bb_ops_create)");
    const int n = ops->neq, np = ops->np;
    const size_t ld = size_t(N_OFFSETS) * np;
    std::vector<double> h(size_t(np) * ld, 0.0);
    for (int o = 0; o < N_OFFSETS; ++o) {
      const int r = lv->m2l_rank[o];
      if (r == 0) continue;
      FMMB_CHECK(lv->m2l_a[o], ERR_INVALID_ARGUMENT, "missing M2L operator");
      // stored transposed, [40 np x np]: row o np + k holds column k of
      // offset o's operator (the M2L row GEMM's W)
      if (r < 0) {  // dense [n x n]
        for (int i = 0; i < n; ++i)
          for (int k = 0; k < n; ++k) h[(size_t(o) * np + k) * np + i] = lv->m2l_a[o][size_t(i) * n + k];
      } else {  // the truncated operator M2 . M1 ([n x r] . [r x n]), as the reference applies it
        FMMB_CHECK(r <= n && lv->m2l_b[o], ERR_INVALID_ARGUMENT, "bad M2L factors");
        for (int i = 0; i < n; ++i)
          for (int k = 0; k < n; ++k) {
            double acc = 0.0;
            for (int q = 0; q < r; ++q) acc += lv->m2l_a[o][size_t(i) * r + q] * lv->m2l_b[o][size_t(q) * n + k];
            h[(size_t(o) * np + k) * np + i] = acc;
          }
      }
    }
    auto e = std::make_unique<LevelEntry>();
    e->dev = LevelOpsDev{};
    e->dev.inv_w = 1.0 / lv->width;
    e->bb_m2l.alloc(h.size(), 0);
    FMMB_CUDA(cudaMemcpy(e->bb_m2l.get(), h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    if (np <= FMM_BB_MAX_RANK)  // the KIFMM's M2L takes the operators as they are
      bb_fragments(*e, np, lv->m2l_rank, [&](int o, int k, int i) {
        return h[(size_t(o) * np + k) * np + i];
      });
    e->dev_copy.alloc(1, 0);
    FMMB_CUDA(cudaMemcpy(e->dev_copy.get(), &e->dev, sizeof(LevelOpsDev), cudaMemcpyHostToDevice));
    ops->levels.push_back(std::move(e));
    *level_id = int(ops->levels.size()) - 1;
  });
}

int fmm_bb_ops_set_basis(fmm_ops *ops, int level_id, int rank, const double *q,
                         const double *const *core) {
  return guarded([&] {
    FMMB_CHECK(ops && q && core, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(ops->method == METHOD_BBFMM, ERR_INVALID_ARGUMENT,
               "fmm_bb_ops_set_basis needs a black-box operator set");
    FMMB_CHECK(level_id >= 0 && level_id < (int)ops->levels.size(), ERR_INVALID_ARGUMENT,
               "unknown operator entry");
    FMMB_CHECK(rank >= 1 && rank <= FMM_BB_MAX_RANK, ERR_INVALID_ARGUMENT,
               "basis rank must be in [1, 64]");
    const int n = ops->neq, np = ops->np, R = FMM_BB_MAX_RANK;
    FMMB_CHECK(np > R, ERR_INVALID_ARGUMENT, "operators this small need no basis");
    LevelEntry &e = *ops->levels[level_id];
    FMMB_CHECK(!e.bb_fast, ERR_INVALID_ARGUMENT, "this width has a basis already");
    std::vector<double> h(size_t(2) * np * R, 0.0);
    for (int i = 0; i < n; ++i)
      for (int k = 0; k < rank; ++k) {
        h[size_t(i) * R + k] = q[size_t(i) * rank + k];
        h[size_t(np) * R + size_t(k) * np + i] = q[size_t(i) * rank + k];
      }
    e.bb_q.alloc(h.size(), 0);
    FMMB_CUDA(cudaMemcpy(e.bb_q.get(), h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    int present[N_OFFSETS];
    for (int o = 0; o < N_OFFSETS; ++o) present[o] = core[o] ? 1 : 0;
    bb_fragments(e, R, present, [&](int o, int k, int i) {
      return i < rank && k < rank ? core[o][size_t(i) * rank + k] : 0.0;
    });
    FMMB_CUDA(cudaMemcpy(e.dev_copy.get(), &e.dev, sizeof(LevelOpsDev), cudaMemcpyHostToDevice));
  });
}

int fmm_kernel_table_create(const double *coef, int j0, int n_octaves, int n_cheb, int *table_id) {
  return guarded([&] {
    FMMB_CHECK(coef && table_id, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(n_octaves >= 1 && n_octaves <= 2048 && n_cheb >= 1 && n_cheb <= 64, ERR_INVALID_ARGUMENT,
               "table size out of range");
    FMMB_CHECK(j0 >= -1000 && j0 + n_octaves <= 1000, ERR_INVALID_ARGUMENT, "octave range out of range");
    auto t = std::make_unique<RadialTable>();
    t->j0 = j0;
    t->noct = n_octaves;
    t->ncheb = n_cheb;
    t->coef.assign(coef, coef + size_t(n_octaves) * n_cheb);
    for (double v : t->coef) FMMB_CHECK(std::isfinite(v), ERR_INVALID_ARGUMENT, "non-finite coefficient");
    std::lock_guard<std::mutex> g(g_tables_mu);
    g_tables.push_back(std::move(t));
    *table_id = int(g_tables.size()) - 1;
  });
}

int fmm_stokes_ops_create(int nequiv, fmm_ops **out) {
  return guarded([&] {
    FMMB_CHECK(out, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(nequiv >= 1 && nequiv <= FMM_MAX_NEQUIV, ERR_INVALID_ARGUMENT, "nequiv must be in [1, 64]");
    auto o = std::make_unique<fmm_ops>();
    o->kernel_id = -1;
    o->kp = KernelParams{};
    o->neq = nequiv;
    o->np = pad8(2 * nequiv + 1);
    o->method = METHOD_STOKES;
    *out = o.release();
  });
}

int fmm_stokes_ops_add(fmm_ops *ops, const fmm_stokes_level_ops *lv, int *level_id) {
  return guarded([&] {
    FMMB_CHECK(ops && lv && level_id && lv->m2l_rank, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(ops->method == METHOD_STOKES, ERR_INVALID_ARGUMENT,
               "fmm_stokes_ops_add needs a Stokes operator set (fmm_stokes_ops_create)");
    const int neq = ops->neq, n1 = 2 * neq + 1, n2 = 2 * neq, np = ops->np;
    const size_t sq = size_t(np) * np, ld = size_t(N_OFFSETS) * np;
    std::vector<double> h;
    auto take = [&](size_t count) {
      size_t at = h.size();
      h.resize(at + ((count + 1) & ~size_t(1)), 0.0);  // 16-byte aligned blocks
      return at;
    };
    const size_t o_lx = take(neq), o_ly = take(neq);
    const size_t o_eu = take(sq), o_ev = take(sq), o_cu = take(sq), o_cv = take(sq);
    const size_t o_mm = take(4 * sq), o_ll = take(4 * sq), o_m2l = take(size_t(np) * ld);
    for (int k = 0; k < neq; ++k) {
      h[o_lx + k] = lv->large_x[k];
      h[o_ly + k] = lv->large_y[k];
    }
    // x = (b . U) . (diag(1/S) VH); the C2E solve drops the extra unknown (column n2)
    auto solve = [&](const double *u, const double *sinv, const double *vh, size_t ou, size_t ov,
                     bool drop_extra) {
      pack_fragments(np, np, [&](int i, int j) {
        return i < n1 && j < n1 ? u[size_t(i) * n1 + j] : 0.0;
      }, h.data() + ou);
      pack_fragments(np, np, [&](int i, int j) {
        return i < n1 && j < n1 && !(drop_extra && j == n2) ? sinv[i] * vh[size_t(i) * n1 + j] : 0.0;
      }, h.data() + ov);
    };
    solve(lv->e2c_u, lv->e2c_sinv, lv->e2c_vh, o_eu, o_ev, false);
    solve(lv->c2e_u, lv->c2e_sinv, lv->c2e_vh, o_cu, o_cv, true);
    pack_fragments(4 * np, np, [&](int ck, int i) {
      const int c = ck / np, k = ck % np;
      return i < n1 && k < n2 ? lv->m2mc[size_t(i) * 4 * n2 + c * n2 + k] : 0.0;
    }, h.data() + o_mm);
    pack_fragments(np, 4 * np, [&](int k, int ci) {
      const int c = ci / np, i = ci % np;
      return i < n1 && k < n2 ? lv->l2lc[size_t(c * n1 + i) * n2 + k] : 0.0;
    }, h.data() + o_ll);
    const bool frag = np <= ST_M2L_NP;
    auto e = std::make_unique<LevelEntry>();
    e->dev = LevelOpsDev{};
    std::vector<double> dense(sq);  // one operator, transposed [np x np]
    for (int o = 0; o < N_OFFSETS; ++o) {
      const int r = lv->m2l_rank[o];
      if (r == 0) continue;
      FMMB_CHECK(lv->m2l_a[o], ERR_INVALID_ARGUMENT, "missing M2L operator");
      FMMB_CHECK(r < 0 || lv->m2l_b[o], ERR_INVALID_ARGUMENT, "bad M2L factors");
      std::fill(dense.begin(), dense.end(), 0.0);
      for (int i = 0; i < n1; ++i)
        for (int k = 0; k < n2; ++k) {
          double v;
          if (r < 0) {
            v = lv->m2l_a[o][size_t(i) * n2 + k];
          } else {  // M2 [n1 x r] . M1 [r x n2], the reference's truncated operator
            v = 0.0;
            for (int q = 0; q < r; ++q) v += lv->m2l_a[o][size_t(i) * r + q] * lv->m2l_b[o][size_t(q) * n2 + k];
          }
          dense[size_t(k) * np + i] = v;
        }
      e->dev.kind[o] = M2L_DENSE;
      if (frag)
        pack_fragments(np, np, [&](int k, int i) { return dense[size_t(k) * np + i]; },
                       h.data() + o_m2l + o * sq);
      else
        std::copy(dense.begin(), dense.end(), h.begin() + o_m2l + o * sq);
    }
    e->st.alloc(h.size(), 0);
    FMMB_CUDA(cudaMemcpy(e->st.get(), h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    double *b = e->st.get();
    auto f2 = [&](size_t o) { return reinterpret_cast<const double2 *>(b + o); };
    e->st_lev = StokesArgs::Level{b + o_lx, b + o_ly, f2(o_eu), f2(o_ev), f2(o_cu), f2(o_cv),
                                  f2(o_mm), f2(o_ll), b + o_m2l};
    for (int o = 0; frag && o < N_OFFSETS; ++o)
      if (e->dev.kind[o] != M2L_NULL) e->dev.m2l_f[o] = f2(o_m2l + o * sq);
    e->dev.inv_w = 1.0 / lv->width;
    e->dev_copy.alloc(1, 0);
    FMMB_CUDA(cudaMemcpy(e->dev_copy.get(), &e->dev, sizeof(LevelOpsDev), cudaMemcpyHostToDevice));
    ops->levels.push_back(std::move(e));
    *level_id = int(ops->levels.size()) - 1;
  });
}

int fmm_ops_destroy(fmm_ops *ops) {
  return guarded([&] {
    if (!ops) return;
    cudaDeviceSynchronize();
    delete ops;
  });
}

// the tree's host-side level offsets: build_tree returns before they arrive
static void tree_ready(fmm_plan *p) {
  if (p) finalize_tree(p->th);
}

int fmm_plan_create(fmm_ops *ops, const double *x, const double *y, int64_t n, int ncutoff,
                    const double *bbox, void *stream, fmm_plan **out) {
  return guarded([&] {
    FMMB_CHECK(ops && x && y && bbox && out, ERR_INVALID_ARGUMENT, "NULL argument");
    retain_pool_memory();
    auto p = std::make_unique<fmm_plan>();
    p->ops = ops;
    p->stream = (cudaStream_t)stream;
    {
      PhaseTimer timer(PH_TREE, p->stream);
      build_tree(p->td, p->th, x, y, n, ncutoff, bbox, p->stream);
    }
    p->bound.assign(p->th.L, -1);
    *out = p.release();
  });
}

int fmm_plan_info(fmm_plan *p, int *n_levels, double *widths, int *n_nodes) {
  return guarded([&] {
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    if (n_nodes) tree_ready(p);  // level counts need the finished tree; L and widths do not
    if (n_levels) *n_levels = p->th.L;
    for (int m = 0; m < p->th.L; ++m) {
      if (widths) widths[m] = p->th.width[m];
      if (n_nodes) n_nodes[m] = p->th.off[m + 1] - p->th.off[m];
    }
  });
}

int fmm_plan_set_precision(fmm_plan *p, int precision) {
  return guarded([&] {
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CHECK(precision == PREC_FP64 || precision == PREC_MIXED, ERR_INVALID_ARGUMENT,
               "precision must be FMM_PRECISION_FP64 or FMM_PRECISION_MIXED");
    FMMB_CHECK(precision == PREC_FP64 || kernel_mixed(p->ops->kernel_id), ERR_UNSUPPORTED,
               "the mixed form needs a kernel with an FP32 form (Laplace, modified Helmholtz)");
    FMMB_CHECK(precision == PREC_FP64 || p->ops->method == METHOD_KIFMM, ERR_UNSUPPORTED,
               "the black-box and Stokes FMMs have an FP64 form only");
    p->precision = precision;
    p->have_expansions = false;
  });
}

int fmm_plan_bind(fmm_plan *p, int level, int level_id) {
  return guarded([&] {
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CHECK(level >= 0 && level < p->th.L, ERR_INVALID_ARGUMENT, "level out of range");
    FMMB_CHECK(level_id >= 0 && level_id < (int)p->ops->levels.size(), ERR_INVALID_ARGUMENT,
               "unknown operator entry");
    p->bound[level] = level_id;
  });
}

int fmm_plan_bind_levels(fmm_plan *p, int n_levels, const int *level_ids) {
  return guarded([&] {
    FMMB_CHECK(p && (level_ids || n_levels == 0), ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(n_levels >= 0 && n_levels <= p->th.L, ERR_INVALID_ARGUMENT, "level count out of range");
    for (int m = 0; m < n_levels; ++m)
      FMMB_CHECK(level_ids[m] >= -1 && level_ids[m] < (int)p->ops->levels.size(),
                 ERR_INVALID_ARGUMENT, "unknown operator entry");
    for (int m = 0; m < n_levels; ++m) p->bound[m] = level_ids[m];
  });
}

static PassArgs pass_args(fmm_plan *p) {
  PassArgs a;
  a.kernel_id = p->ops->kernel_id;
  a.kp = p->ops->kp;
  a.neq = p->ops->neq;
  a.np = p->ops->np;
  a.td = &p->td;
  a.th = &p->th;
  a.ops_dev = p->ops_dev.get();
  a.sync = p->sync.get();
  if (p->precision == PREC_FP64) a.fail = p->pass_fail();
  if (p->has_dipoles) {
    a.dvx = p->dvx.get();
    a.dvy = p->dvy.get();
  }
  return a;
}

__global__ void k_gather_dipoles(const double *__restrict__ str, const double *__restrict__ nx,
                                 const double *__restrict__ ny, const int *__restrict__ ordv,
                                 int64_t n, double *__restrict__ dvx, double *__restrict__ dvy) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int o = ordv[i];
    dvx[i] = str[o] * nx[o];
    dvy[i] = str[o] * ny[o];
  }
}

// The plan's per-level operator table, gathered on the device from the
// operator set's entries (no host copy: the launch arguments carry the
// entries' addresses)
struct LevelOpsSrc {
  const LevelOpsDev *p[FMM_MAX_LEVELS_DEV];
  double width[FMM_MAX_LEVELS_DEV];  // what a box's sources keep to; infinite once they were moved
  // scaling of levels without operators (0 and 1 need none: no expansions there,
  // but the mixed near field of a leaf there does read its scaling)
  double inv_w[FMM_MAX_LEVELS_DEV], kofs[FMM_MAX_LEVELS_DEV];
};
static_assert(sizeof(LevelOpsDev) % sizeof(int) == 0, "LevelOpsDev is copied as words");
static_assert(offsetof(LevelOpsDev, kofs) == offsetof(LevelOpsDev, inv_w) + sizeof(double),
              "k_gather_level_ops fills in both together");

__global__ void k_gather_level_ops(LevelOpsSrc src, LevelOpsDev *__restrict__ dst) {
  constexpr int NW = int(sizeof(LevelOpsDev) / sizeof(int));
  const int *from = reinterpret_cast<const int *>(src.p[blockIdx.x]);
  int *to = reinterpret_cast<int *>(dst + blockIdx.x);
  constexpr int SCALE = int(offsetof(LevelOpsDev, inv_w) / sizeof(int));
  constexpr int BOX = int(offsetof(LevelOpsDev, box32) / sizeof(int));
  const double iw = from ? src.p[blockIdx.x]->inv_w : src.inv_w[blockIdx.x];
  for (int i = threadIdx.x; i < NW; i += blockDim.x) to[i] = from ? from[i] : 0;
  // what the tree adds, each word by the thread that has just copied it
  auto mine = [](int word) { return threadIdx.x == word % blockDim.x; };
  if (mine(BOX)) to[BOX] = __float_as_int(float(src.width[blockIdx.x] * iw));
  if (!from)
    for (int k = 0; k < 4; ++k)
      if (mine(SCALE + k)) {
        const double d = k < 2 ? iw : src.kofs[blockIdx.x];
        to[SCALE + k] = k & 1 ? __double2hiint(d) : __double2loint(d);
      }
}

static void upload_level_ops(fmm_plan *p, cudaStream_t s) {
  const int L = p->th.L;
  FMMB_CHECK(L <= FMM_MAX_LEVELS_DEV, ERR_INVALID_ARGUMENT, "too many levels");
  p->ops_dev.alloc(L, s);
  LevelOpsSrc src{};
  const bool scaled = p->ops->method == METHOD_KIFMM && kernel_scaled(p->ops->kernel_id);
  for (int m = 0; m < L; ++m) {
    const double w = p->th.width[m];
    src.width[m] = p->moved ? HUGE_VAL : w;
    if (p->bound[m] >= 0) {
      src.p[m] = p->ops->levels[p->bound[m]]->dev_copy.get();
    } else {
      src.inv_w[m] = scaled ? 1.0 / w : 1.0;
      src.kofs[m] = scaled ? kernel_offset(p->ops->kernel_id, p->ops->kp, w) : 0.0;
    }
  }
  k_gather_level_ops<<<L, 128, 0, s>>>(src, p->ops_dev.get());
  FMMB_CUDA(cudaGetLastError());
}

static StokesArgs stokes_args(fmm_plan *p, cudaStream_t) {
  StokesArgs a{};
  a.neq = p->ops->neq;
  a.np = p->ops->np;
  a.td = &p->td;
  a.th = &p->th;
  a.ops_dev = p->ops_dev.get();
  for (int m = 0; m < p->th.L && m < FMM_MAX_LEVELS_DEV; ++m)
    if (p->bound[m] >= 0) a.lev[m] = p->ops->levels[p->bound[m]]->st_lev;
  if (p->has_st_dipoles) {
    const size_t n = size_t(p->th.n_points);
    double *d = p->st_dip.get();
    a.sgx = d;
    a.sgy = d + n;
    a.dnx = d + 2 * n;
    a.dny = d + 3 * n;
  }
  return a;
}

static BBArgs bb_args(fmm_plan *p, cudaStream_t) {
  BBArgs b{};
  b.kernel_id = p->ops->kernel_id;
  b.kp = p->ops->kp;
  b.p = p->ops->p;
  b.np = p->ops->np;
  b.td = &p->td;
  b.th = &p->th;
  b.m2mc = p->ops->bb_m2mc.get();
  b.m2mct = p->ops->bb_m2mct.get();
  if (const double *sep = p->ops->bb_sep.get()) {
    b.m2m_sep = sep;
    b.l2l_sep = sep + p->ops->bb_sep.n / 2;
  }
  b.any_fast = false;
  for (int m = 0; m < p->th.L && m < FMM_MAX_LEVELS_DEV; ++m) {
    const LevelEntry *e = p->bound[m] >= 0 ? p->ops->levels[p->bound[m]].get() : nullptr;
    b.m2l_cat[m] = e ? e->bb_m2l.get() : nullptr;
    b.q[m] = e ? e->bb_q.get() : nullptr;
    b.fast[m] = m >= 2 && e && e->bb_fast;
    b.any_fast = b.any_fast || b.fast[m];
  }
  b.ops_dev = p->ops_dev.get();
  return b;
}

static void build_stokes(fmm_plan *p, const double *fx, const double *fy, const double *sgx,
                         const double *sgy, const double *nx, const double *ny, void *stream);

int fmm_build_expansions2(fmm_plan *p, const double *fx, const double *fy, void *stream) {
  return guarded([&] { build_stokes(p, fx, fy, nullptr, nullptr, nullptr, nullptr, stream); });
}

int fmm_build_expansions2_dipole(fmm_plan *p, const double *fx, const double *fy,
                                 const double *sigma_x, const double *sigma_y, const double *dip_nx,
                                 const double *dip_ny, void *stream) {
  return guarded([&] {
    FMMB_CHECK(sigma_x && sigma_y && dip_nx && dip_ny, ERR_INVALID_ARGUMENT, "NULL argument");
    build_stokes(p, fx, fy, sigma_x, sigma_y, dip_nx, dip_ny, stream);
  });
}

static void build_stokes(fmm_plan *p, const double *fx, const double *fy, const double *sgx,
                         const double *sgy, const double *nx, const double *ny, void *stream) {
  {
    tree_ready(p);
    FMMB_CHECK(p && fx && fy, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(p->ops->method == METHOD_STOKES, ERR_INVALID_ARGUMENT,
               "fmm_build_expansions2 takes Stokes plans (two force components)");
    cudaStream_t s = (cudaStream_t)stream;
    p->has_st_dipoles = sgx != nullptr;
    if (sgx) {  // stresslet strengths and normals in the tree's order
      const int64_t n = p->th.n_points;
      p->st_dip.alloc(4 * size_t(n), s);
      const double *src[4] = {sgx, sgy, nx, ny};
      for (int c = 0; c < 4; ++c) gather_sorted(src[c], p->td.ordv.get(), n, p->st_dip.get() + c * n, s);
    }
    const TreeHost &th = p->th;
    for (int m = 2; m < th.L; ++m)
      FMMB_CHECK(p->bound[m] >= 0, ERR_NOT_READY, "operators not bound for every level >= 2");
    const int np = p->ops->np;
    const int64_t total = th.n_total();
    upload_level_ops(p, s);
    StokesArgs a = stokes_args(p, s);
    p->tau_s.alloc(th.n_points, s);
    p->tau2_s.alloc(th.n_points, s);
    gather_sorted(fx, p->td.ordv.get(), th.n_points, p->tau_s.get(), s);
    gather_sorted(fy, p->td.ordv.get(), th.n_points, p->tau2_s.get(), s);
    ZeroBatch zb(s);
    for (DevBuf<double> *b : {&p->partial, &p->mult, &p->ple, &p->loc}) {
      b->alloc(total * np, s);
      zb.add(*b);
    }
    zb.run();
    run_stokes_upward(a, p->tau_s.get(), p->tau2_s.get(), p->partial.get(), p->mult.get(), s);
    run_stokes_downward(a, p->mult.get(), p->ple.get(), p->loc.get(), s);
    p->have_expansions = true;
  }
}

int fmm_build_expansions_multi(fmm_plan *p, const double *tau, int n_rhs, int64_t ld_tau,
                               void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p && tau, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(p->ops->method == METHOD_KIFMM && p->precision == PREC_FP64, ERR_UNSUPPORTED,
               "several charge columns: FP64 KIFMM plans");
    const TreeHost &th = p->th;
    FMMB_CHECK(n_rhs >= 1 && ld_tau >= th.n_points, ERR_INVALID_ARGUMENT, "bad n_rhs or ld_tau");
    cudaStream_t s = (cudaStream_t)stream;
    for (int m = 2; m < th.L; ++m)
      FMMB_CHECK(p->bound[m] >= 0, ERR_NOT_READY, "operators not bound for every level >= 2");
    const int np = p->ops->np;
    const int64_t total = th.n_total(), n = th.n_points, cs = total * np;
    upload_level_ops(p, s);
    p->has_dipoles = false;
    p->sync.alloc(3, s);
    PassArgs a = pass_args(p);
    p->tau_s.alloc((size_t)n_rhs * n, s);
    p->mult.alloc((size_t)n_rhs * cs, s);
    p->ple.alloc((size_t)n_rhs * cs, s);
    p->loc.alloc((size_t)n_rhs * cs, s);
    ZeroBatch zb(s);
    zb.add(p->mult).add(p->ple).add(p->loc).add(p->sync);
    zb.run();
    gather_sorted(tau, p->td.ordv.get(), n, p->tau_s.get(), s, n_rhs, ld_tau);
    // every pass once for all columns
    run_upward(a, p->tau_s.get(), p->mult.get(), s, n_rhs, n, cs);
    run_m2l(a, p->mult.get(), p->ple.get(), s, n_rhs, cs);
    run_downward(a, p->ple.get(), p->loc.get(), s, n_rhs, cs);
    p->n_rhs = n_rhs;
    p->ready_recorded = false;  // the split evaluation serves single-column builds
    p->have_expansions = true;
  });
}

int fmm_evaluate_multi(fmm_plan *p, const double *tx, const double *ty, int64_t m, int check,
                       double *out, int64_t ld_out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CHECK(p->have_expansions, ERR_NOT_READY, "build_expansions has not run");
    FMMB_CHECK(p->ops->method == METHOD_KIFMM && p->precision == PREC_FP64, ERR_UNSUPPORTED,
               "several charge columns: FP64 KIFMM plans");
    FMMB_CHECK(m >= 0 && ld_out >= m, ERR_INVALID_ARGUMENT, "bad target count or ld_out");
    if (m == 0) return;
    FMMB_CHECK(tx && ty && out, ERR_INVALID_ARGUMENT, "NULL argument");
    cudaStream_t s = (cudaStream_t)stream;
    PassArgs a = pass_args(p);
    a.ops_dev = p->ops_dev.get();
    DevBuf<uint64_t> tkeys;
    DevBuf<int> tperm;
    DevBuf<double> txs, tys;
    {
      PhaseTimer timer(PH_SORT_TGT, s);
      txs.alloc(m, s);
      tys.alloc(m, s);
      sort_points(tx, ty, m, p->th, tkeys, tperm, s, p->th.L > 1 ? p->th.L - 1 : 1, txs.get(),
                  tys.get(), p->td.sort_fail.get());
    }
    run_evaluate_multi(a, p->tau_s.get(), p->th.n_points, p->n_rhs, p->loc.get(),
                       (int64_t)p->th.n_total() * p->ops->np, txs.get(), tys.get(), tkeys.get(),
                       tperm.get(), m, check, out, ld_out, s);
  });
}

int fmm_evaluate_sources_multi(fmm_plan *p, int check, double *out, int64_t ld_out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CHECK(p->have_expansions, ERR_NOT_READY, "build_expansions has not run");
    FMMB_CHECK(p->ops->method == METHOD_KIFMM && p->precision == PREC_FP64, ERR_UNSUPPORTED,
               "several charge columns: FP64 KIFMM plans");
    FMMB_CHECK(out && ld_out >= p->th.n_points, ERR_INVALID_ARGUMENT, "NULL out or ld_out too small");
    cudaStream_t s = (cudaStream_t)stream;
    PassArgs a = pass_args(p);
    a.ops_dev = p->ops_dev.get();
    const TreeDev &td = p->td;
    run_evaluate_multi(a, p->tau_s.get(), p->th.n_points, p->n_rhs, p->loc.get(),
                       (int64_t)p->th.n_total() * p->ops->np, td.sx.get(), td.sy.get(),
                       td.pkeys.get(), td.ordv.get(), p->th.n_points, check, out, ld_out, s);
  });
}

int fmm_plan_create_local(fmm_ops *ops, const double *x, const double *y, int64_t n, int ncutoff,
                          double min_width, const double *bbox, void *stream, fmm_plan **out) {
  return guarded([&] {
    FMMB_CHECK(ops && x && y && bbox && out, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(ops->method == METHOD_KIFMM && ops->kernel_id >= 0, ERR_INVALID_ARGUMENT,
               "a local plan takes a kernel operator set (fmm_ops_create)");
    FMMB_CHECK(min_width >= 0.0, ERR_INVALID_ARGUMENT, "negative minimum width");
    // a box of level m (width w0 / 2^m, halved level by level as the
    // reference does) splits only while its width exceeds 2 min_width
    const double w0 = bbox[1] - bbox[0];
    int max_split = 0;
    for (double w = w0; max_split < 64 && w > 2.0 * min_width; w *= 0.5) ++max_split;
    retain_pool_memory();
    auto p = std::make_unique<fmm_plan>();
    p->ops = ops;
    p->stream = (cudaStream_t)stream;
    {
      PhaseTimer timer(PH_TREE, p->stream);
      build_tree(p->td, p->th, x, y, n, ncutoff, bbox, p->stream, max_split);
    }
    p->bound.assign(p->th.L, -1);
    *out = p.release();
  });
}

int fmm_local_evaluate(fmm_plan *p, const double *tau, const double *tx, const double *ty,
                       int64_t m, int check, const int64_t *src_cat, const int64_t *tgt_cat,
                       double *out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p && tau, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(p->ops->method == METHOD_KIFMM, ERR_INVALID_ARGUMENT, "not a local plan");
    FMMB_CHECK((src_cat == nullptr) == (tgt_cat == nullptr), ERR_INVALID_ARGUMENT,
               "source and target categories go together");
    FMMB_CHECK(m >= 0, ERR_INVALID_ARGUMENT, "negative target count");
    if (m == 0) return;
    FMMB_CHECK(tx && ty && out, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(m < (int64_t(1) << 31) - 1, ERR_INVALID_ARGUMENT, "more than 2^31-2 targets");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t n = p->th.n_points;
    p->tau_s.alloc(n, s);
    gather_sorted(tau, p->td.ordv.get(), n, p->tau_s.get(), s);
    DevBuf<int64_t> scat;
    if (src_cat) {
      scat.alloc(n, s);
      gather_sorted_i64(src_cat, p->td.ordv.get(), n, scat.get(), s);
    }
    PassArgs a = pass_args(p);
    DevBuf<uint64_t> tkeys;
    DevBuf<int> tperm;
    DevBuf<double> txs, tys;
    {
      PhaseTimer timer(PH_SORT_TGT, s);
      txs.alloc(m, s);
      tys.alloc(m, s);
      sort_points(tx, ty, m, p->th, tkeys, tperm, s, p->th.L > 1 ? p->th.L - 1 : 1, txs.get(),
                  tys.get(), p->td.sort_fail.get());
    }
    run_local_evaluate(a, p->tau_s.get(), txs.get(), tys.get(), tkeys.get(), tperm.get(), m,
                       check, src_cat ? scat.get() : nullptr, tgt_cat, out, s);
  });
}

static void build_expansions_impl(fmm_plan *p, const double *tau, void *stream);

int fmm_build_expansions(fmm_plan *p, const double *tau, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p && tau, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(p->ops->method != METHOD_STOKES, ERR_INVALID_ARGUMENT,
               "Stokes plans take fmm_build_expansions2 (two force components)");
    p->has_dipoles = false;
    build_expansions_impl(p, tau, stream);
  });
}

int fmm_build_expansions_dipole(fmm_plan *p, const double *tau, const double *dip_str,
                                const double *dip_nx, const double *dip_ny, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p && dip_str && dip_nx && dip_ny, ERR_INVALID_ARGUMENT, "NULL argument");
    FMMB_CHECK(p->ops->method == METHOD_KIFMM && p->ops->kernel_id == KERNEL_LAPLACE,
               ERR_UNSUPPORTED, "dipole sources: KIFMM plans of the Laplace kernel");
    FMMB_CHECK(p->precision == PREC_FP64, ERR_UNSUPPORTED, "dipole sources: FP64 form only");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t n = p->th.n_points;
    p->dvx.alloc(n, s);
    p->dvy.alloc(n, s);
    if (n > 0) {
      k_gather_dipoles<<<grid_for(n, 256), 256, 0, s>>>(dip_str, dip_nx, dip_ny,
                                                         p->td.ordv.get(), n, p->dvx.get(),
                                                         p->dvy.get());
      FMMB_CUDA(cudaGetLastError());
    }
    p->has_dipoles = true;
    build_expansions_impl(p, tau, stream);
  });
}

// the build itself (FP64 / mixed KIFMM or black-box), after the entry's checks;
// tau = NULL: zero charges
static void build_expansions_impl(fmm_plan *p, const double *tau, void *stream) {
  {
    p->n_rhs = 1;
    cudaStream_t s = (cudaStream_t)stream;
    const TreeHost &th = p->th;
    for (int m = 2; m < th.L; ++m)
      FMMB_CHECK(p->bound[m] >= 0, ERR_NOT_READY, "operators not bound for every level >= 2");
    const int np = p->ops->np;
    const int64_t total = th.n_total();
    if (p->ops->method == METHOD_BBFMM) {
      upload_level_ops(p, s);
      BBArgs b = bb_args(p, s);
      p->tau_s.alloc(th.n_points, s);
      gather_sorted(tau, p->td.ordv.get(), th.n_points, p->tau_s.get(), s);
      p->mult.alloc(total * np, s);
      p->ple.alloc(total * np, s);
      const bool basis = b.any_fast && np > FMM_BB_MAX_RANK;
      if (basis) {
        p->partial.alloc(total * FMM_BB_MAX_RANK, s);
        p->loc.alloc(total * FMM_BB_MAX_RANK, s);
      }
      ZeroBatch zb(s);
      zb.add(p->mult).add(p->ple);
      if (basis) zb.add(p->loc);  // (the M2L writes the rows of real groups only)
      zb.run();
      run_bb_upward(b, p->tau_s.get(), p->mult.get(), s);
      run_bb_downward(b, p->mult.get(), p->ple.get(), basis ? p->partial.get() : nullptr,
                      basis ? p->loc.get() : nullptr, s);
      p->have_expansions = true;
      return;
    }
    std::unique_ptr<PhaseTimer> t_prep(new PhaseTimer(PH_PREP, s));
    upload_level_ops(p, s);
    split_prepare(p);
    p->ready_recorded = false;
    split_scratch_prepare(p, s);
    p->sync.alloc(3, s);
    PassArgs a = pass_args(p);
    p->tau_s.alloc(th.n_points, s);
    if (tau)
      gather_sorted(tau, p->td.ordv.get(), th.n_points, p->tau_s.get(), s);
    else
      p->tau_s.zero(s);
    p->ple.alloc(total * np, s);
    if (p->precision == PREC_MIXED) {
      p->mult32.alloc(total * np, s);
      p->loc32.alloc(total * np, s);
      p->msum.alloc(total, s);
      p->lsum.alloc(total, s);
      p->mult_tc.alloc(total * 2 * np, s);
      // a split near field (if evaluation splits) runs beside the upward and
      // downward passes and pauses while the M2L runs: hold clear now, set
      // before the M2L; m2l_done recorded after it
      p->hold_armed = split_enabled(PREC_MIXED);
      if (p->hold_armed) p->near_hold.alloc(1, s);
      p->err.alloc(2, s);  // [0] error flag, [1] M2L tile counter
      ZeroBatch zb(s);
      zb.add(p->ple).add(p->mult32).add(p->mult_tc).add(p->loc32).add(p->msum).add(p->lsum).add(p->err);
      if (p->hold_armed) zb.add(p->near_hold);
      zb.run();
      p->tsum.alloc(total, s);
      node_charge_sums(a, p->tau_s.get(), p->tsum.get(), s);
      // sorted charges and box charge sums are all the near field reads
      FMMB_CUDA(cudaEventRecord(p->ev_ready, s));
      p->ready_recorded = true;
      t_prep.reset();
      run_upward_mixed(a, p->tau_s.get(), p->tsum.get(), p->mult32.get(), p->msum.get(),
                       p->mult_tc.get(), s);
      if (p->hold_armed) FMMB_CUDA(cudaMemsetAsync(p->near_hold.get(), 1, 1, s));
      run_m2l_mixed(a, p->mult32.get(), p->mult_tc.get(), p->msum.get(), p->ple.get(),
                    p->err.get(), s);
      if (p->hold_armed) FMMB_CUDA(cudaEventRecord(p->ev_m2l, s));
      run_downward_mixed(a, p->ple.get(), p->loc32.get(), p->lsum.get(), s);
    } else {
      p->mult.alloc(total * np, s);
      p->loc.alloc(total * np, s);
      ZeroBatch(s).add(p->ple).add(p->mult).add(p->loc).add(p->sync).run();
      FMMB_CUDA(cudaEventRecord(p->ev_ready, s));  // sorted charges: all the near field reads
      p->ready_recorded = true;
      t_prep.reset();
      PassStream ps(p, s);
      run_upward(a, p->tau_s.get(), p->mult.get(), ps.stream());
      run_m2l(a, p->mult.get(), p->ple.get(), ps.stream());
      run_downward(a, p->ple.get(), p->loc.get(), ps.stream());
      ps.join();
    }
    p->have_expansions = true;
  }
}

namespace {
// outputs of an evaluator id (FMM_EVAL_*)
int evaluator_outputs(int evaluator) {
  FMMB_CHECK(evaluator == FMM_EVAL_POTENTIAL || evaluator == FMM_EVAL_GRADIENT ||
                 evaluator == FMM_EVAL_STOKES,
             ERR_INVALID_ARGUMENT, "evaluator must be one of FMM_EVAL_POTENTIAL, _GRADIENT, _STOKES");
  return evaluator == FMM_EVAL_POTENTIAL ? 1 : 3;
}

// a plan's method accepts the evaluator (Stokes plans: (u, v, p) only)
void check_evaluator(fmm_plan *p, int evaluator) {
  FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
  const bool st = p->ops->method == METHOD_STOKES;
  FMMB_CHECK(st == (evaluator == FMM_EVAL_STOKES), ERR_INVALID_ARGUMENT,
             st ? "Stokes plans evaluate FMM_EVAL_STOKES (u, v, p)"
                : "FMM_EVAL_STOKES needs a Stokes plan");
}

void evaluate_points(fmm_plan *p, int nout, const double *tx, const double *ty, int64_t m,
                     int check, double *out, int64_t ld_out, cudaStream_t s) {
  FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
  FMMB_CHECK(p->have_expansions, ERR_NOT_READY, "build_expansions has not run");
  FMMB_CHECK(m >= 0, ERR_INVALID_ARGUMENT, "negative target count");
  if (m == 0) return;
  FMMB_CHECK(tx && ty && out, ERR_INVALID_ARGUMENT, "NULL argument");
  FMMB_CHECK(m < (int64_t(1) << 31) - 1, ERR_INVALID_ARGUMENT, "more than 2^31-2 targets");
  FMMB_CHECK(nout == 1 || ld_out >= m, ERR_INVALID_ARGUMENT, "ld_out is smaller than the target count");
  PassArgs a = pass_args(p);
  DevBuf<uint64_t> tkeys;
  DevBuf<int> tperm;
  DevBuf<double> txs, tys;
  txs.alloc(m, s);
  tys.alloc(m, s);
  if (p->ops->method == METHOD_KIFMM) {
    split_note(p, false);
    // targets binned into their leaves (a descent along each key's digits and
    // a count per leaf) instead of sorted
    EvalItems it;
    {
      PhaseTimer timer(PH_SORT_TGT, s);
      tperm.alloc(m, s);
      eval_items_binned(a, tx, ty, m, it, txs.get(), tys.get(), tperm.get(), s);
    }
    if (p->precision == PREC_MIXED)
      run_evaluate_mixed(a, p->tau_s.get(), p->tsum.get(), p->loc32.get(), p->lsum.get(), txs.get(),
                         tys.get(), nullptr, tperm.get(), m, check, nout, out, ld_out, s, &it);
    else
      run_evaluate(a, p->tau_s.get(), p->loc.get(), txs.get(), tys.get(), nullptr, tperm.get(), m,
                   check, nout, out, ld_out, s, &it);
    return;
  }
  // evaluator ids carry the output count; Stokes plans produce (u, v, p)
  {
    PhaseTimer timer(PH_SORT_TGT, s);
    // leaves live on levels <= L-1: their first L-1 digits decide everything
    sort_points(tx, ty, m, p->th, tkeys, tperm, s, p->th.L > 1 ? p->th.L - 1 : 1, txs.get(),
                tys.get(), p->td.sort_fail.get());
  }
  if (p->ops->method == METHOD_STOKES)
    run_stokes_evaluate(stokes_args(p, s), p->tau_s.get(), p->tau2_s.get(), p->loc.get(), txs.get(),
                        tys.get(), tkeys.get(), tperm.get(), m, check, out, ld_out, s);
  else if (p->ops->method == METHOD_BBFMM)
    run_bb_evaluate(bb_args(p, s), p->tau_s.get(), p->ple.get(), txs.get(), tys.get(), tkeys.get(),
                    tperm.get(), m, check, nout, out, ld_out, s);
  else if (p->precision == PREC_MIXED)
    run_evaluate_mixed(a, p->tau_s.get(), p->tsum.get(), p->loc32.get(), p->lsum.get(), txs.get(),
                       tys.get(), tkeys.get(), tperm.get(), m, check, nout, out, ld_out, s);
  else
    run_evaluate(a, p->tau_s.get(), p->loc.get(), txs.get(), tys.get(), tkeys.get(), tperm.get(),
                 m, check, nout, out, ld_out, s);
}


void evaluate_own_sources(fmm_plan *p, int nout, int check, double *out, int64_t ld_out,
                          cudaStream_t s) {
  FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
  FMMB_CHECK(p->have_expansions, ERR_NOT_READY, "build_expansions has not run");
  FMMB_CHECK(out, ERR_INVALID_ARGUMENT, "NULL argument");
  const TreeDev &td = p->td;
  const int64_t m = p->th.n_points;
  FMMB_CHECK(nout == 1 || ld_out >= m, ERR_INVALID_ARGUMENT, "ld_out is smaller than the source count");
  PassArgs a = pass_args(p);
  // the tree's sorted copy: keys sorted on at least their top L-1 digits,
  // which is all that leaf location reads
  if (p->ops->method == METHOD_STOKES)
    run_stokes_evaluate(stokes_args(p, s), p->tau_s.get(), p->tau2_s.get(), p->loc.get(),
                        td.sx.get(), td.sy.get(), td.pkeys.get(), td.ordv.get(), m, check, out,
                        ld_out, s);
  else if (p->ops->method == METHOD_BBFMM)
    run_bb_evaluate(bb_args(p, s), p->tau_s.get(), p->ple.get(), td.sx.get(), td.sy.get(),
                    td.pkeys.get(), td.ordv.get(), m, check, nout, out, ld_out, s);
  else if (nout == 1 && p->ready_recorded && p->n_rhs == 1 && split_enabled(p->precision)) {
    // near field on the side stream, started when the charges were sorted
    split_note(p, true);
    SplitEval se{p->side, p->ev_ready, p->ev_near, p->ev_far};
    if (p->split_scratch_ready && !capturing(s)) se.scratch = &p->split_scratch;
    if (p->precision == PREC_MIXED && p->hold_armed) {
      se.hold = p->near_hold.get();
      se.m2l_done = p->ev_m2l;
    }
    if (p->precision == PREC_MIXED)
      run_evaluate_sources_split_mixed(a, p->tau_s.get(), p->tsum.get(), p->loc32.get(),
                                       p->lsum.get(), check, out, s, se);
    else
      run_evaluate_sources_split(a, p->tau_s.get(), p->loc.get(), check, out, s, se);
  } else {
    split_note(p, false);
    if (p->precision == PREC_MIXED)
      run_evaluate_mixed(a, p->tau_s.get(), p->tsum.get(), p->loc32.get(), p->lsum.get(),
                         td.sx.get(), td.sy.get(), td.pkeys.get(), td.ordv.get(), m, check, nout,
                         out, ld_out, s);
    else
      run_evaluate(a, p->tau_s.get(), p->loc.get(), td.sx.get(), td.sy.get(), td.pkeys.get(),
                   td.ordv.get(), m, check, nout, out, ld_out, s);
  }
}
}  // namespace

int fmm_evaluate(fmm_plan *p, const double *tx, const double *ty, int64_t m, int check,
                 double *out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    check_evaluator(p, FMM_EVAL_POTENTIAL);
    evaluate_points(p, 1, tx, ty, m, check, out, m, (cudaStream_t)stream);
  });
}

int fmm_evaluate_sources(fmm_plan *p, int check, double *out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    check_evaluator(p, FMM_EVAL_POTENTIAL);
    evaluate_own_sources(p, 1, check, out, 0, (cudaStream_t)stream);
  });
}

int fmm_evaluate_outputs(fmm_plan *p, int evaluator, const double *tx, const double *ty,
                         int64_t m, int check, double *out, int64_t ld_out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    const int nout = evaluator_outputs(evaluator);
    check_evaluator(p, evaluator);
    evaluate_points(p, nout, tx, ty, m, check, out, ld_out, (cudaStream_t)stream);
  });
}

int fmm_evaluate_sources_outputs(fmm_plan *p, int evaluator, int check, double *out,
                                 int64_t ld_out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    const int nout = evaluator_outputs(evaluator);
    check_evaluator(p, evaluator);
    evaluate_own_sources(p, nout, check, out, ld_out, (cudaStream_t)stream);
  });
}

int fmm_plan_status(fmm_plan *p) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CUDA(cudaStreamSynchronize(p->stream));
    FMMB_CUDA(cudaGetLastError());
    if (p->err.get()) {
      int h = 0;
      FMMB_CUDA(cudaMemcpy(&h, p->err.get(), sizeof(int), cudaMemcpyDeviceToHost));
      FMMB_CHECK(h == 0, ERR_CUDA, "a tensor-core wait ran out of time; results are invalid");
    }
    if (p->td.sort_fail.get()) {
      int h = 0;
      FMMB_CUDA(cudaMemcpy(&h, p->td.sort_fail.get(), sizeof(int), cudaMemcpyDeviceToHost));
      FMMB_CHECK(h == 0, ERR_CUDA,
                 "a sort's or scan's grid barrier wait ran out of time; results are invalid");
    }
    if (p->precision == PREC_FP64 && p->pass_fail()) {
      int h = 0;
      FMMB_CUDA(cudaMemcpy(&h, p->pass_fail(), sizeof(int), cudaMemcpyDeviceToHost));
      FMMB_CHECK(h == 0, ERR_CUDA,
                 "a level pass's wait (grid barrier or operator copy) ran out of time; results are "
                 "invalid (NaN)");
    }
  });
}

int fmm_diag_fail_passes(fmm_plan *p, void *stream) {
  return guarded([&] {
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CHECK(p->have_expansions && p->precision == PREC_FP64 && p->pass_fail(), ERR_NOT_READY,
               "no FP64 KIFMM expansions have been built");
    FMMB_CUDA(cudaMemsetAsync(p->pass_fail(), 1, sizeof(int), (cudaStream_t)stream));
  });
}

int fmm_plan_drop_expansions(fmm_plan *p) {
  return guarded([&] {
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    // device memory returns to the pool in the plan stream's order
    p->tau_s.release();
    p->tau2_s.release();
    p->mult.release();
    p->ple.release();
    p->loc.release();
    p->mult32.release();
    p->loc32.release();
    p->mult_tc.release();
    p->msum.release();
    p->lsum.release();
    p->tsum.release();
    p->partial.release();
    p->dvx.release();
    p->dvy.release();
    p->has_dipoles = false;
    p->st_dip.release();
    p->has_st_dipoles = false;
    p->split_scratch.release();
    p->split_scratch_ready = false;
    p->have_expansions = false;
    p->ready_recorded = false;
  });
}

int fmm_plan_move_sources(fmm_plan *p, const double *x, const double *y, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    const int64_t n = p->th.n_points;
    if (n == 0) return;
    FMMB_CHECK(x && y, ERR_INVALID_ARGUMENT, "NULL argument");
    cudaStream_t s = (cudaStream_t)stream;
    // the tree's sorted copy, in the tree's own order (sorted -> original)
    gather_sorted(x, p->td.ordv.get(), n, p->td.sx.get(), s);
    gather_sorted(y, p->td.ordv.get(), n, p->td.sy.get(), s);
    p->moved = true;
    p->have_expansions = false;
    p->ready_recorded = false;
  });
}

int fmm_plan_destroy(fmm_plan *p) {
  // no host wait: the plan's device buffers go back to the pool with
  // cudaFreeAsync on the stream they were allocated on, after the work
  // already queued there
  return guarded([&] { delete p; });
}

int fmm_tree_export(fmm_plan *p, double *xmin, double *ymin, int *bot, int *top, int *parent,
                    int *child, uint8_t *flags, int *coll, int *il, int *ordv) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    const size_t T = p->th.n_total();
    cudaStream_t s = p->stream;
    auto cp = [&](void *dst, const void *src, size_t bytes) {
      if (dst && bytes) FMMB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
    };
    cp(xmin, p->td.xmin.get(), T * sizeof(double));
    cp(ymin, p->td.ymin.get(), T * sizeof(double));
    cp(bot, p->td.bot.get(), T * sizeof(int));
    cp(top, p->td.top.get(), T * sizeof(int));
    cp(parent, p->td.parent.get(), T * sizeof(int));
    cp(child, p->td.child.get(), T * sizeof(int));
    cp(flags, p->td.flags.get(), T * sizeof(uint8_t));
    cp(coll, p->td.coll.get(), T * 9 * sizeof(int));
    cp(il, p->td.il.get(), T * N_OFFSETS * sizeof(int));
    cp(ordv, p->td.ordv.get(), size_t(p->th.n_points) * sizeof(int));
    FMMB_CUDA(cudaStreamSynchronize(s));
  });
}

int fmm_direct(int kernel_id, const double *kparams, const double *sx, const double *sy,
               const double *tau, int64_t ns, const double *tx, const double *ty, int64_t nt,
               int check, double *out, void *stream) {
  return guarded([&] {
    FMMB_CHECK(kernel_known(kernel_id), ERR_UNSUPPORTED, "unknown kernel id");
    FMMB_CHECK(ns >= 0 && nt >= 0, ERR_INVALID_ARGUMENT, "negative size");
    if (nt == 0) return;
    FMMB_CHECK(tx && ty && out && (ns == 0 || (sx && sy && tau)), ERR_INVALID_ARGUMENT,
               "NULL argument");
    const KernelParams kp = kernel_params(kernel_id, kparams);
    run_direct(kernel_id, kp, sx, sy, tau, ns, tx, ty, nt, check, out, (cudaStream_t)stream);
  });
}

int fmm_diag_log2(const double *x, int64_t n, double *out_table, double *out_library,
                  void *stream) {
  return guarded([&] {
    FMMB_CHECK(n >= 0, ERR_INVALID_ARGUMENT, "negative size");
    if (n == 0) return;
    FMMB_CHECK(x && out_table && out_library, ERR_INVALID_ARGUMENT, "NULL argument");
    run_diag_log2(x, n, out_table, out_library, (cudaStream_t)stream);
  });
}

int fmm_set_split_evaluation(int mode) {
  return guarded([&] {
    FMMB_CHECK(mode >= -1 && mode <= 1, ERR_INVALID_ARGUMENT, "mode must be -1, 0 or 1");
    if (mode == -1) {
      const char *e = getenv("FLEXMM_B200_SPLIT_EVAL");
      mode = e ? (e[0] == '0' ? 0 : 1) : -1;
    }
    g_split_mode.store(mode);
  });
}

int fmm_timing_enable(int on) {
  return guarded([&] {
    auto &R = TimingRegistry::get();
    std::lock_guard<std::mutex> g(R.mu);
    R.enabled = on != 0;
  });
}

int fmm_timing_read(double *ms, int64_t *launches) {
  return guarded([&] {
    auto &R = TimingRegistry::get();
    std::lock_guard<std::mutex> g(R.mu);
    for (int i = 0; i < FMM_N_PHASES; ++i) {
      if (ms) ms[i] = 0.0;
      if (launches) launches[i] = 0;
    }
    for (auto &r : R.recs) {
      FMMB_CUDA(cudaEventSynchronize(r.b));
      float t = 0.f;
      FMMB_CUDA(cudaEventElapsedTime(&t, r.a, r.b));
      if (ms) ms[r.phase] += t;
      if (launches) launches[r.phase] += 1;
      R.pool.push_back(r.a);
      R.pool.push_back(r.b);
    }
    R.recs.clear();
  });
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free evaluation.
//
// fmm_evaluate_noalloc does the work of fmm_evaluate without allocating
// device memory: its scratch (target keys and permutation, sorted target
// coordinates, per-node target ranges, sort and scan workspace) lives in the
// file-scope array below.  The array is part of the library image, so every
// GPU that loads the library holds it (NOALLOC_SCRATCH_BYTES) until the
// process exits.  Every call shares it and it keeps the last call's contents;
// nothing in it needs to start at zero (every scratch word is written before
// it is read).  Calls that overlap on the GPU (two streams, two threads) race
// on it and must be serialised by the caller.
namespace {
constexpr size_t NOALLOC_SCRATCH_BYTES = size_t(24) << 20;  // 24 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

// device address of the array, looked up once per device (with it current) by
// the first call on that device; that first call should come before any
// stream capture
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mu;
void *g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};

void *noalloc_scratch_for_current_device() {
  int dev = 0;
  FMMB_CUDA(cudaGetDevice(&dev));
  FMMB_CHECK(dev >= 0 && dev < NOALLOC_MAX_DEVICES, ERR_UNSUPPORTED, "device ordinal too large");
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void *ptr = nullptr;
    FMMB_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    g_noalloc_ptr[dev] = ptr;
  }
  return g_noalloc_ptr[dev];
}

size_t round256(size_t b) { return (b + 255) & ~size_t(255); }
}  // namespace

extern "C" int fmm_evaluate_noalloc(fmm_plan *p, const double *tx, const double *ty, int64_t m,
                                    int check, double *out, void *stream) {
  return guarded([&] {
    tree_ready(p);
    FMMB_CHECK(p, ERR_INVALID_ARGUMENT, "plan is NULL");
    FMMB_CHECK(p->have_expansions, ERR_NOT_READY, "build_expansions has not run");
    FMMB_CHECK(p->precision == PREC_FP64, ERR_UNSUPPORTED,
               "fmm_evaluate_noalloc evaluates FP64 plans only");
    FMMB_CHECK(p->ops->method == METHOD_KIFMM, ERR_UNSUPPORTED,
               "fmm_evaluate_noalloc evaluates KIFMM plans only");
    FMMB_CHECK(!p->has_dipoles, ERR_UNSUPPORTED,
               "fmm_evaluate_noalloc evaluates charge sources only (no dipoles)");
    FMMB_CHECK(m >= 0, ERR_INVALID_ARGUMENT, "negative target count");
    FMMB_CHECK(m <= FMM_NOALLOC_MAX_TARGETS, ERR_CAPACITY,
               "fmm_evaluate_noalloc: more than FMM_NOALLOC_MAX_TARGETS targets");
    const int total = p->th.n_total();
    FMMB_CHECK(total <= FMM_NOALLOC_MAX_NODES, ERR_CAPACITY,
               "fmm_evaluate_noalloc: tree has more than FMM_NOALLOC_MAX_NODES nodes");
    if (m == 0) return;
    FMMB_CHECK(tx && ty && out, ERR_INVALID_ARGUMENT, "NULL argument");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned char *base = static_cast<unsigned char *>(noalloc_scratch_for_current_device());
    // carve the scratch
    const int digits = p->th.L > 1 ? p->th.L - 1 : 1;
    const size_t sort_bytes = round256(sort_points_scratch_bytes(m, digits));
    size_t at = 0;
    auto carve = [&](size_t bytes) {
      unsigned char *q = base + at;
      at += round256(bytes);
      return q;
    };
    uint64_t *tkeys = (uint64_t *)carve(m * sizeof(uint64_t));
    int *tperm = (int *)carve(m * sizeof(int));
    double *txs = (double *)carve(m * sizeof(double));
    double *tys = (double *)carve(m * sizeof(double));
    int4 *items = (int4 *)carve((total + m / EVAL_CHUNK + 1) * sizeof(int4));
    int *n_items = (int *)carve((1 + EVAL_COUNTERS) * sizeof(int));
    void *sort_tmp = carve(sort_bytes);
    FMMB_CHECK(at <= NOALLOC_SCRATCH_BYTES, ERR_CAPACITY,
               "fmm_evaluate_noalloc: scratch needs exceed the static array");
    // the same passes as fmm_evaluate, on the static scratch
    const PassArgs a = pass_args(p);
    {
      PhaseTimer timer(PH_SORT_TGT, s);
      sort_points_scratch(tx, ty, m, p->th, digits, tkeys, tperm, txs, tys, sort_tmp, sort_bytes,
                          p->td.sort_fail.get(), s);
    }
    run_evaluate_scratch(a, p->tau_s.get(), p->loc.get(), txs, tys, tkeys, tperm, m, check, out,
                         items, n_items, s);
  });
}
