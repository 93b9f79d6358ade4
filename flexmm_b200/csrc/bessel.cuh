// Modified Bessel functions K0 and K1 in FP64 for the modified Helmholtz
// kernel K0(k r) / (2 pi) (examples/kifmm_modified_helmholtz.py:25-39; its
// gradient uses K1, examples/pure_kifmm_modified_helmholtz_gradient.py:45-70).
//
// The reference evaluates K0 through piecewise Chebyshev tables fitted to
// scipy.special.k0 (function_generator, examples/kifmm_modified_helmholtz.py:28).
// Here, likewise tabulated but built without a third-party library, as
// functions of s = x^2 (the kernels have the squared distance at hand):
//  * x < 1: the ascending series (Abramowitz & Stegun 9.6.13 and 9.6.11) in
//    y = x^2/4 <= 1/4, as polynomials,
//      K0 = -(ln(x/2) + gamma) I0(x) + sum_k H_k y^k / (k!)^2,
//      K1 / x = 1/x^2 + ((ln(x/2) + gamma) i1(y) - (1/2) sum_k (H_k + H_(k+1)) y^k / (k!(k+1)!)) / 2,
//    i1(y) = sum_k y^k / (k!(k+1)!), H_k the harmonic numbers, cut where the
//    next term is below 1e-17 of the sum; ln x = (ln 2 / 2) log2 s, from the
//    passes' table-driven log2 or CUDA's;
//  * 1 <= x < 1024: h_0(x) = e^x K0(x) and h_1(x) = e^x K1(x) / x as polynomials
//    of degree 10 in x - c on each eighth of the octaves [2^j, 2^(j+1)),
//    j = 0..9 (c the middle).  The coefficients are computed on the host
//    (bessel_table_host() in capi.cu) from the integral representations
//    e^x K0(x) = int_0^inf exp(-2x sinh^2(t/2)) dt,
//    e^x K1(x) = int_0^inf exp(-2x sinh^2(t/2)) cosh t dt, by the trapezoidal
//    rule (exponentially convergent for these analytic integrands);
//  * x >= 1024: 0 (below the smallest double).
// Bound by the FP64 pipe.  x < 1 takes about 33 FP64 instructions; the series
// summed term by term with a division in each, before, took about 250, and the
// tables' degree-19 Clenshaw recurrence about 90 where a degree-10 polynomial
// with its square root and exponential takes about 50.  The potential step at
// 200k clustered points, k = 10: step 2.73 -> 1.00 ms (evaluation kernels 0.42 ms), S2M 258 ->
// 65 us; 0.86 ms and 46 us with the later changes to S2M, tree and scratch.  Largest relative error over x in [1e-6, 300]: 6e-16 (before: 7e-16
// below x = 1, 4e-15 above).
#pragma once
#include <math.h>

namespace fmmb {

constexpr int BESSEL_OCTAVES = 10;  // [1, 2) ... [512, 1024)
constexpr int BESSEL_PARTS = 8;     // equal intervals of an octave
constexpr int BESSEL_INTERVALS = BESSEL_OCTAVES * BESSEL_PARTS;
constexpr int BESSEL_NCOEF = 11;    // coefficients of an interval's polynomial
constexpr int BESSEL_ROW = 12;      // their row in the table (16-byte aligned)
// table layout: [function n = 0, 1][interval][BESSEL_ROW]
constexpr int BESSEL_TABLE_DOUBLES = 2 * BESSEL_INTERVALS * BESSEL_ROW;
constexpr double EULER_GAMMA = 0.57721566490153286061;

// K0(x) and, with K1 = true, K1(x) / x, for 0 < x < 1: s = x^2, l2 = log2(s)
template <bool K1>
__device__ __forceinline__ void bessel_small(double s, double l2, double &k0, double &k1x) {
  constexpr double LN2 = 0.69314718055994530942;
  const double y = 0.25 * s;
  // -(ln(x/2) + gamma)
  const double m = fma(l2, -0.5 * LN2, LN2 - EULER_GAMMA);
  // 1 / (k!)^2 and H_k / (k!)^2 (numerators and denominators exact)
  double i0 = 1.0 / 1625702400.0, s0 = 7129.0 / (2520.0 * 131681894400.0);
  i0 = fma(i0, y, 1.0 / 25401600.0);
  s0 = fma(s0, y, 761.0 / (280.0 * 1625702400.0));
  i0 = fma(i0, y, 1.0 / 518400.0);
  s0 = fma(s0, y, 363.0 / (140.0 * 25401600.0));
  i0 = fma(i0, y, 1.0 / 14400.0);
  s0 = fma(s0, y, 49.0 / (20.0 * 518400.0));
  i0 = fma(i0, y, 1.0 / 576.0);
  s0 = fma(s0, y, 137.0 / (60.0 * 14400.0));
  i0 = fma(i0, y, 1.0 / 36.0);
  s0 = fma(s0, y, 25.0 / (12.0 * 576.0));
  i0 = fma(i0, y, 1.0 / 4.0);
  s0 = fma(s0, y, 11.0 / (6.0 * 36.0));
  i0 = fma(i0, y, 1.0);
  s0 = fma(s0, y, 3.0 / (2.0 * 4.0));
  i0 = fma(i0, y, 1.0);
  s0 = fma(s0, y, 1.0);
  k0 = fma(m, i0, s0 * y);
  if (K1) {
    // 1 / (k!(k+1)!) and (H_k + H_(k+1)) / (k!(k+1)!)
    double i1 = 1.0 / 14631321600.0, h1 = (761.0 / 280.0 + 7129.0 / 2520.0) / 14631321600.0;
    i1 = fma(i1, y, 1.0 / 203212800.0);
    h1 = fma(h1, y, (363.0 / 140.0 + 761.0 / 280.0) / 203212800.0);
    i1 = fma(i1, y, 1.0 / 3628800.0);
    h1 = fma(h1, y, (49.0 / 20.0 + 363.0 / 140.0) / 3628800.0);
    i1 = fma(i1, y, 1.0 / 86400.0);
    h1 = fma(h1, y, (137.0 / 60.0 + 49.0 / 20.0) / 86400.0);
    i1 = fma(i1, y, 1.0 / 2880.0);
    h1 = fma(h1, y, (25.0 / 12.0 + 137.0 / 60.0) / 2880.0);
    i1 = fma(i1, y, 1.0 / 144.0);
    h1 = fma(h1, y, (11.0 / 6.0 + 25.0 / 12.0) / 144.0);
    i1 = fma(i1, y, 1.0 / 12.0);
    h1 = fma(h1, y, (3.0 / 2.0 + 11.0 / 6.0) / 12.0);
    i1 = fma(i1, y, 1.0 / 2.0);
    h1 = fma(h1, y, (1.0 + 3.0 / 2.0) / 2.0);
    i1 = fma(i1, y, 1.0);
    h1 = fma(h1, y, 1.0);
    k1x = fma(-0.5, fma(m, i1, 0.5 * h1), 1.0 / s);
  }
}

// K0(x) and, with K1 = true, K1(x) / x, for 1 <= x < 1024.  Not inlined: one
// copy serves a sweep's unrolled pairs.
template <bool K1>
__device__ __noinline__ double2 bessel_large(double x, const double *__restrict__ tab) {
  const int hi = __double2hiint(x);
  // interval from the exponent and the top three mantissa bits; its middle
  const int iv = min(max((hi >> 17) - (1023 << 3), 0), BESSEL_INTERVALS - 1);
  const double d = x - __hiloint2double((hi & ~0x1FFFF) | 0x10000, 0);
  const double w = exp(-x);
  double r[2] = {0.0, 0.0};
#pragma unroll
  for (int n = 0; n < (K1 ? 2 : 1); ++n) {
    const double2 *c =
        reinterpret_cast<const double2 *>(tab + (n * BESSEL_INTERVALS + iv) * BESSEL_ROW);
    double p = __ldg(c + 5).x;
#pragma unroll
    for (int i = 4; i >= 0; --i) {
      const double2 q = __ldg(c + i);
      p = fma(fma(p, d, q.y), d, q.x);
    }
    r[n] = p * w;
  }
  return make_double2(r[0], r[1]);
}

// k^2 as the arguments s = k^2 r^2 take it: 0 where the square has lost bits
// below the normal range (every pair then goes by bessel_any's last branch)
__host__ __device__ __forceinline__ double bessel_k2(double k) {
  const double k2 = k * k;
  return k2 < 0x1p-1022 ? 0.0 : k2;
}

// K0(x) and, with K1 = true, k^2 K1(x) / x (the gradient's factor, 1 / r^2 for
// small x), for any x = k r >= 0: r2 = r^2, s = bessel_k2(k) r2
template <bool K1>
__device__ __noinline__ double2 bessel_any(double k, double r2, double s,
                                           const double *__restrict__ tab) {
  double2 r = make_double2(0.0, 0.0);
  if (s >= 1.0 && s < 1048576.0) {
    r = bessel_large<K1>(sqrt(s), tab);
  } else if (s >= 0x1p-1022 && s < 1.0) {
    bessel_small<K1>(s, log2(s), r.x, r.y);
  } else {
    // a square leaves the range: the distance itself may not
    const double x = k * sqrt(r2);
    if (x < 1.0) {
      bessel_small<K1>(x * x, 2.0 * log2(x), r.x, r.y);
      // (x K1(x) = 1 + O(x^2 log x): 1 to the last bit)
      if (K1 && x < 0x1p-30) return make_double2(r.x, 1.0 / r2);
    } else if (x < 1024.0) {
      r = bessel_large<K1>(x, tab);
    } else {
      r.x = r.y = x >= 1024.0 ? 0.0 : x;  // NaN stays
    }
  }
  if (K1) r.y = k * (k * r.y);  // (k^2 may leave the range where this does not)
  return r;
}

}  // namespace fmmb
