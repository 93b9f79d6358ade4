// Device kernel functors, registered under the reference's example names.
//
//   Laplace_Eval: -log(|t-s|^2) / (4 pi)       examples/kifmm_laplace.py:24-29
//   Modified_Helmholtz_Eval: K0(k |t-s|) / (2 pi)  examples/kifmm_modified_helmholtz.py:33-39
//   a tabulated radial kernel f(|t-s|), as the reference's examples build
//   with function_generator (e.g. the Struve kernel, examples/bbfmm_struve.py:29-46)
//
// A functor evaluates K(source, target) for source (sx, sy) and target
// (tx, ty); the FMM kernels are templated on it, so the functor inlines into
// every loop the way the reference's numba kernel inlines into its closures
// (flexmm/flexmm2d/helpers.py:87-151).
#pragma once
#include <math.h>

#include <cfloat>
#include <cmath>

#include "bessel.cuh"
#include "common.cuh"
#include "log2_table.cuh"

namespace fmmb {

enum KernelId : int { KERNEL_LAPLACE = 0, KERNEL_MOD_HELMHOLTZ = 1, KERNEL_RADIAL_TABLE = 2 };

// the caller's parameters (p[0] = helmholtz k for the modified Helmholtz
// kernel) and the device's Bessel tables (bessel.cuh)
struct KernelParams {
  double p[4];
  const double *table;
};

// ---------------------------------------------------------------------------
// Table-driven FP64 log2, after P. T. P. Tang, "Table-driven implementation
// of the logarithm function in IEEE floating-point arithmetic", ACM TOMS 16
// (1990): d = 2^e m, m in [1, 2); F = 1 + j/256 is the table point nearest m
// and c next to 1/F, so r = m c - 1 (one fused multiply-add) has |r| <= 2^-9 and
//   log2 d = e - log2 c + log2(1 + r),  log2(1 + r) = r q(r),
// q the degree-4 polynomial that takes log2(1 + r)/r's values at the five
// Chebyshev nodes of [-2^-9, 2^-9] (error of r q(r): 9e-19).  The table holds c
// and -log2 c for j = 0..256 (log2_table.cuh), copied to shared memory by each
// block; its values are doubles to 2^-13 of their last place.  So the error is
// the two roundings of the last sum, half an ulp each: at most 2.2e-16 relative
// to max(1, |log2 d|), 2e-18 next to d = 1, in 9 FP64 instructions.  Zero,
// subnormal, infinite and NaN arguments take the library log2 instead.
// 257 rows and not 129: with these q would have to have one more term (an FP64
// instruction in 13 of a pair) or be off by 5e-17, more than all else next to
// d = 1.  Copied and not formed in each block by a division and a logarithm a
// row: a step of 1M clustered points, near field 1.2 ms of it, takes 2254 us with 129
// rows copied, 2285 with 129 formed, 2282 with 257 copied, 2319 with 257 formed,
// 2286 with 129 copied and the longer q.
struct Log2Table {
  double2 t[LOG2_TAB_N + 1];
  __device__ void fill() {
    for (int i = threadIdx.x; i <= LOG2_TAB_N; i += blockDim.x) t[i] = LOG2_ROWS[i];
  }
};

// log2_rare_key(d) >= LOG2_RARE for arguments outside the table path: zero,
// subnormal, negative, infinite or NaN (one unsigned compare; the largest key
// of several arguments tests them together)
constexpr unsigned LOG2_RARE = 0x7FE00000u;
__device__ __forceinline__ unsigned log2_rare_key(double d) {
  return (unsigned)(__double2hiint(d) - 0x00100000);
}
__device__ __forceinline__ bool log2_tab_rare(double d) { return log2_rare_key(d) >= LOG2_RARE; }

// log2 of a positive normal finite d (callers route log2_tab_rare arguments
// elsewhere)
__device__ __forceinline__ double log2_tab(double d, const double2 *__restrict__ tab) {
  constexpr double Q0 = 0x1.71547652b82fep+0, Q1 = -0x1.71547652b5c85p-1,
                   Q2 = 0x1.ec709dc39c20ap-2, Q3 = -0x1.7154c3445f43cp-2,
                   Q4 = 0x1.27770702adfd1p-2;
  const int hi = __double2hiint(d), lo = __double2loint(d);
  const int mh = hi & 0x000FFFFF;
  const double m = __hiloint2double(mh | 0x3FF00000, lo);  // [1, 2)
  const double2 tj = tab[(mh + (1 << 11)) >> 12];          // nearest 1/256 step: 0..256
  const double r = fma(m, tj.x, -1.0);
  // the exponent as a double without a conversion instruction: the bits
  // (0x43300000, n) are 2^52 + n
  const double e = __hiloint2double(0x43300000, hi >> 20) - (4503599627370496.0 + 1023.0);
  double q = fma(r, Q4, Q3);
  q = fma(r, q, Q2);
  q = fma(r, q, Q1);
  q = fma(r, q, Q0);
  return fma(r, q, e + tj.y);
}

// 1/d for d in [2^-1022, 2^1021): the hardware's approximate reciprocal
// (rcp.approx.ftz.f64, about 20 bits), refined by the third-order Newton step
// y (1 + e + e^2), e = 1 - d y: error e^3, below the last bit.  (Above,
// 1/d comes down to 2^-1022, below which the approximation is flushed to 0.)
constexpr unsigned RCP_RARE = 0x7FB00000u;  // log2_rare_key from here on: not for rcp_newton
__device__ __forceinline__ double rcp_newton(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// Shared-memory state a functor needs inside a kernel (the log2 table of
// LaplaceF64T); empty for the other functors.  bind() is called by every
// thread of the block before the functor's first use.
template <class KF, bool = KF::kLogTable>
struct FunctorSmem {
  __device__ void bind(KF &) {}
};

struct LaplaceF64 {
  static constexpr bool kLogTable = false;
  __host__ __device__ explicit LaplaceF64(const KernelParams &) {}
  __device__ __forceinline__ double operator()(double sx, double sy, double tx, double ty) const {
    const double dx = tx - sx, dy = ty - sy;
    return -log(dx * dx + dy * dy) * (1.0 / (4.0 * M_PI));
  }
  // potential and its gradient in the target position, times q, added to
  // (u, ux, uy) (Gradient_Eval, examples/pure_kifmm_laplace_gradient.py:32-55)
  __device__ __forceinline__ void grad(double sx, double sy, double tx, double ty, double q,
                                       double &u, double &ux, double &uy) const {
    const double dx = tx - sx, dy = ty - sy, d2 = dx * dx + dy * dy;
    const double s = -(1.0 / (2.0 * M_PI)) / d2 * q;
    u += -log(d2) * (1.0 / (4.0 * M_PI)) * q;
    ux += s * dx;
    uy += s * dy;
  }
};

// The Laplace kernel of the FP64 passes: LaplaceF64 with the table-driven
// log2 above.  raw(dx, dy) = log2(dx^2 + dy^2), so K = kFold * raw; the P2P
// and L2T loops fold kFold into their staged charges / locals.
// A table functor's pair loops split raw into arg() of the squared distance,
// at() of an argument inside the table path, and raw_rare() for the others.
struct LaplaceF64T {
  static constexpr bool kLogTable = true;
  static constexpr unsigned kRare = LOG2_RARE;  // arguments with this key or above: raw_rare
  static constexpr double kFold = -0.69314718055994530942 / (4.0 * M_PI);  // -ln2 / (4 pi)
  const double2 *lt = nullptr;  // the block's table (FunctorSmem::bind)
  __host__ __device__ explicit LaplaceF64T(const KernelParams &) {}
  __device__ __forceinline__ double arg(double d2) const { return d2; }
  __device__ __forceinline__ double at(double s) const { return log2_tab(s, lt); }
  // a pair whose argument is outside the table path
  __device__ __forceinline__ double raw_rare(double dx, double dy) const {
    return log2(fma(dy, dy, dx * dx));
  }
  __device__ __forceinline__ double raw(double dx, double dy) const {
    const double s = arg(fma(dy, dy, dx * dx));
    return log2_tab_rare(s) ? raw_rare(dx, dy) : at(s);
  }
  __device__ __forceinline__ double operator()(double sx, double sy, double tx, double ty) const {
    return kFold * raw(tx - sx, ty - sy);
  }
  // raw value and raw gradient factor of a pair inside the table path: the
  // potential is kFold * v, its gradient in the target position
  // grad_fold * w * (dx, dy) (Gradient_Eval, examples/pure_kifmm_laplace_gradient.py:32-55)
  static __host__ __device__ double grad_fold(const KernelParams &) { return -1.0 / (2.0 * M_PI); }
  __device__ __forceinline__ void at_grad(double s, double &v, double &w) const {
    v = at(s);
    w = rcp_newton(s);
  }
  __device__ __forceinline__ void grad_rare(double dx, double dy, int check, double &v,
                                            double &w) const {
    v = w = 0.0;
    if (check && dx == 0.0 && dy == 0.0) return;
    const double d2 = fma(dy, dy, dx * dx);
    v = log2(d2);
    w = 1.0 / d2;
  }
};

template <class KF>
struct FunctorSmem<KF, true> {
  Log2Table tab;
  __device__ void bind(KF &k) {
    tab.fill();
    __syncthreads();
    k.lt = tab.t;
  }
};

struct ModHelmholtzF64 {
  static constexpr bool kLogTable = false;
  double k, k2;
  const double *tab;
  __host__ __device__ explicit ModHelmholtzF64(const KernelParams &kp)
      : k(kp.p[0]), k2(bessel_k2(kp.p[0])), tab(kp.table) {}
  __device__ __forceinline__ double operator()(double sx, double sy, double tx, double ty) const {
    const double dx = tx - sx, dy = ty - sy, d2 = dx * dx + dy * dy;
    return bessel_any<false>(k, d2, k2 * d2, tab).x * (1.0 / (2.0 * M_PI));
  }
  // potential and its gradient in the target position, times q:
  // d/dt K0(k r) = -k K1(k r) (t - s) / r
  // (examples/pure_kifmm_modified_helmholtz_gradient.py:45-70)
  __device__ __forceinline__ void grad(double sx, double sy, double tx, double ty, double q,
                                       double &u, double &ux, double &uy) const {
    const double dx = tx - sx, dy = ty - sy, d2 = dx * dx + dy * dy;
    const double2 b = bessel_any<true>(k, d2, k2 * d2, tab);
    const double s = -b.y * (1.0 / (2.0 * M_PI)) * q;
    u += b.x * (1.0 / (2.0 * M_PI)) * q;
    ux += s * dx;
    uy += s * dy;
  }
};

// The modified Helmholtz kernel of the FP64 passes: ModHelmholtzF64 in the
// form of a table functor (see LaplaceF64T), its table path the small
// arguments x < 1 with the table-driven log2.  The line lies at the series'
// end: near-field distances are at most about 2.8 leaf widths, so a sweep is
// on this path unless k is above 1/3 of a reciprocal leaf width.
struct ModHelmholtzF64T {
  static constexpr bool kLogTable = true;
  static constexpr unsigned kRare = 0x3FE00000u;  // log2_rare_key(1.0)
  static constexpr double kFold = 1.0 / (2.0 * M_PI);
  double k, k2;
  const double *tab;
  const double2 *lt = nullptr;
  __host__ __device__ explicit ModHelmholtzF64T(const KernelParams &kp)
      : k(kp.p[0]), k2(bessel_k2(kp.p[0])), tab(kp.table) {}
  static __host__ __device__ double grad_fold(const KernelParams &) { return -1.0 / (2.0 * M_PI); }
  __device__ __forceinline__ double arg(double d2) const { return k2 * d2; }
  __device__ __forceinline__ double at(double s) const {
    double k0, k1x;
    bessel_small<false>(s, log2_tab(s, lt), k0, k1x);
    return k0;
  }
  __device__ __forceinline__ double raw_rare(double dx, double dy) const {
    const double d2 = fma(dy, dy, dx * dx);
    return bessel_any<false>(k, d2, k2 * d2, tab).x;
  }
  __device__ __forceinline__ double raw(double dx, double dy) const {
    const double s = arg(fma(dy, dy, dx * dx));
    return log2_rare_key(s) >= kRare ? raw_rare(dx, dy) : at(s);
  }
  __device__ __forceinline__ double operator()(double sx, double sy, double tx, double ty) const {
    return kFold * raw(tx - sx, ty - sy);
  }
  __device__ __forceinline__ void at_grad(double s, double &v, double &w) const {
    bessel_small<true>(s, log2_tab(s, lt), v, w);
    w *= k2;  // here and not on the sums: 1 / k^2 and with it K1(x) / x may leave the range
  }
  __device__ __forceinline__ void grad_rare(double dx, double dy, int check, double &v,
                                            double &w) const {
    v = w = 0.0;
    if (check && dx == 0.0 && dy == 0.0) return;
    const double d2 = fma(dy, dy, dx * dx);
    const double2 b = bessel_any<true>(k, d2, k2 * d2, tab);
    v = b.x;
    w = b.y;
  }
};

// K(s, t) = f(|t - s|) with f tabulated as Chebyshev series on the octaves
// [2^j, 2^(j+1)), j = j0 .. j0 + noct - 1 (table [noct][ncheb], built on the
// host from any function; the octave grid resolves power-law and log
// behaviour at 0).  Distances outside the tabulated range are clamped to it.
struct RadialTableF64 {
  static constexpr bool kLogTable = false;
  const double2 *tab;  // rows of coefficient pairs (an odd count ends with a zero)
  int j0, npair;
  double lo, hi;
  __host__ __device__ explicit RadialTableF64(const KernelParams &kp)
      : tab(reinterpret_cast<const double2 *>(kp.table)), j0(int(kp.p[1])),
        npair((int(kp.p[3]) + 1) / 2), lo(ldexp(1.0, j0)),
        hi(ldexp(1.0, j0 + int(kp.p[2])) * (1.0 - 1e-16)) {}
  // Bound by the FP64 pipe (24 coefficients: about 75 instructions, sqrt
  // included) and the coefficients' gathers, a pair each.  The octave and the
  // place in it come from the bits: u = (2 r - 3 a) / a with a = 2^(e-1) is
  // 2 m - 3 of the mantissa m in [1, 2), the same number.  Near fields of 140k
  // targets in a table of 24 coefficients: 611 us with frexp, ldexp, the
  // division and single coefficients, 440 so.
  __device__ __forceinline__ double f(double r) const {
    r = fmin(fmax(r, lo), hi);
    const int hw = __double2hiint(r);
    // (normal: tables start at 2^-1000)
    const double m = __hiloint2double((hw & 0xFFFFF) | 0x3FF00000, __double2loint(r));
    const double u = fma(2.0, m, -3.0), u2 = 2.0 * u;
    const double2 *c = tab + ((hw >> 20) - 1023 - j0) * npair;
    double b1 = 0.0, b2 = 0.0;
#pragma unroll 4
    for (int i = npair - 1; i >= 1; --i) {
      const double2 q = __ldg(c + i);
      b2 = fma(u2, b1, -b2) + q.y;
      b1 = fma(u2, b2, -b1) + q.x;
    }
    const double2 q = __ldg(c);
    b2 = fma(u2, b1, -b2) + q.y;
    return fma(u, b2, -b1) + q.x;
  }
  __device__ __forceinline__ double operator()(double sx, double sy, double tx, double ty) const {
    const double dx = tx - sx, dy = ty - sy;
    return f(sqrt(dx * dx + dy * dy));
  }
  // a tabulated kernel carries no derivative table: gradients are not offered
  __device__ __forceinline__ void grad(double, double, double, double, double, double &, double &,
                                       double &) const {}
};

// log2 on the special-function unit, denormal inputs flushed to zero
// (lg2.approx.ftz.f32: relative error ~2^-22 on normal inputs).
__device__ __forceinline__ float lg2_ftz(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// FP32 evaluation for the mixed-precision passes.  The log kernel is scale
// invariant up to a constant, K(w r) = offset(w) + K(r) with offset(w) =
// -log(w^2)/(4 pi): the mixed passes evaluate K in FP32 on coordinates divided
// by the box width (O(1) arguments, so FP32 keeps the kernel's variation to
// ~1e-7 absolute) and add offset(w) times the charge sum in FP64.  Kernels
// without such a decomposition set kScaled = false and offset() = 0.
//
// Radial form used by the P2P loop: K(dx, dy) = kScale * radial(dx^2 + dy^2),
// with kScale folded into the staged charges.  radial() is only called on
// squared distances >= FLT_MIN (smaller ones are coincident pairs, handled
// apart in FP64).
struct LaplaceF32 {
  static constexpr bool kScaled = true;
  static constexpr bool kNearForm = false;
  // radial(d2) is -inf for d2 below FLT_MIN (the flushed log2 of 0)
  static constexpr bool kInfAtZero = true;
  static constexpr float kScale = (float)(-0.69314718055994531 / (4.0 * M_PI));  // -ln2 / (4 pi)
  __host__ __device__ explicit LaplaceF32(const KernelParams &) {}
  // -log(d2)/(4 pi) = -(ln 2 / 4 pi) * log2(d2); on width-scaled coordinates
  // the hardware log2's error is ~2e-7 of log2, ~1e-8 of K
  // (dx, dy) = target - source
  __device__ __forceinline__ float operator()(float dx, float dy) const {
    return lg2_ftz(dx * dx + dy * dy) * kScale;
  }
  __device__ __forceinline__ float radial(float d2) const { return lg2_ftz(d2); }
  // gradient in the target position: kGradScale * (dx, dy) / d2 on width-scaled
  // coordinates (times 1/w for absolute units)
  static constexpr double kGradScale = -1.0 / (2.0 * M_PI);
  static double offset(double w, const KernelParams &) { return -std::log(w * w) / (4.0 * M_PI); }
};

// K0 in FP32 (A&S 9.8.1, 9.8.5, 9.8.6: Abramowitz & Stegun, Handbook of
// Mathematical Functions, polynomial approximations of I0 and K0):
//   x <= 2: K0(x) = -ln(x/2) I0(x) + P(t^2), t = x/2 (|error| < 1e-8), with
//           I0(x) = Q((x/3.75)^2) (relative error < 1.6e-7);
//   x > 2:  K0(x) = exp(-x) / sqrt(x) R(2/x) (relative error < 1.9e-7).
// Both branches are computed and one selected (no divergence within a warp
// of pairs at mixed distances).  K0(0) = +inf (the flushed log of 0).
// bessel_k0_f32_small is the x <= 2 branch alone, for sweeps whose distances
// are known to lie there (the same bits at 24 instructions for 40).
__device__ __forceinline__ float bessel_k0_f32_small(float x) {
  const float y = (x * (1.f / 3.75f)) * (x * (1.f / 3.75f));
  const float i0 = fmaf(y, fmaf(y, fmaf(y, fmaf(y, fmaf(y, fmaf(y, 0.0045813f, 0.0360768f), 0.2659732f),
                                                   1.2067492f), 3.0899424f), 3.5156229f), 1.f);
  const float t2 = 0.25f * x * x;
  const float p = fmaf(t2, fmaf(t2, fmaf(t2, fmaf(t2, fmaf(t2, fmaf(t2, 0.0000074f, 0.0001075f), 0.00262698f),
                                                   0.0348859f), 0.23069756f), 0.4227842f), -0.57721566f);
  // -ln(x/2) = (1 - log2 x) ln 2
  return fmaf((1.f - lg2_ftz(x)) * 0.69314718f, i0, p);
}
__device__ __forceinline__ float bessel_k0_f32(float x) {
  const float small = bessel_k0_f32_small(x);
  const float z = 2.f * __frcp_rn(fmaxf(x, 2.f));
  const float r = fmaf(z, fmaf(z, fmaf(z, fmaf(z, fmaf(z, fmaf(z, 0.00053208f, -0.0025154f), 0.00587872f),
                                                  -0.01062446f), 0.02189568f), -0.07832358f), 1.25331414f);
  const float large = __expf(-x) * rsqrtf(fmaxf(x, 2.f)) * r;
  return x <= 2.f ? small : large;
}

// FP32 evaluation of K0(k r) / (2 pi) for the mixed passes.  K0 has no scale
// decomposition: the passes evaluate it on box-centred coordinates in the
// caller's units (kScaled = false, offset 0); FP32 keeps a pair's distance
// to ~1e-7 of the box width, which bounds the per-pair error as for the log
// kernel on width-scaled coordinates.
struct ModHelmholtzF32 {
  static constexpr bool kScaled = false;
  static constexpr bool kNearForm = true;  // radial_near
  // radial(d2) is +inf for d2 below FLT_MIN (K0 at a flushed 0)
  static constexpr bool kInfAtZero = true;
  static constexpr float kScale = (float)(1.0 / (2.0 * M_PI));
  float k;
  __host__ __device__ explicit ModHelmholtzF32(const KernelParams &kp) : k((float)kp.p[0]) {}
  // (squared distances below FLT_MIN flushed to 0: K0 = +inf there)
  __device__ __forceinline__ float radial(float d2) const {
    return bessel_k0_f32(k * (d2 < FLT_MIN ? 0.f : sqrtf(d2)));
  }
  // radial() of distances with k r <= 2, which near_all() promises of every
  // point within (hx, hy) of this one: the rounded products stay below 2
  __device__ __forceinline__ float radial_near(float d2) const {
    return bessel_k0_f32_small(k * (d2 < FLT_MIN ? 0.f : sqrtf(d2)));
  }
  __device__ __forceinline__ bool near_all(float hx, float hy) const {
    return k * sqrtf(hx * hx + hy * hy) <= 1.9999f;
  }
  // (dx, dy) = target - source
  __device__ __forceinline__ float operator()(float dx, float dy) const {
    return radial(dx * dx + dy * dy) * kScale;
  }
  static double offset(double, const KernelParams &) { return 0.0; }
};

}  // namespace fmmb
