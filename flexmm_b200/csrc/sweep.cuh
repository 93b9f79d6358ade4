// Pair sweeps of charge (and dipole) sources for the evaluation items
// (items.cuh): the near field of the KIFMM and black-box forms, and the KIFMM
// far field (the equivalent sources on the leaf's large circle).
#pragma once
#include "items.cuh"

namespace fmmb {
namespace {

constexpr double INV_2PI = 1.0 / (2.0 * M_PI);

// double-layer kernel of the Laplace kernel -log(r^2)/(4 pi): the field at
// offset (ax, ay) = target - source of a dipole (dx, dy) = strength * normal,
// (d . a) / (2 pi |a|^2) (Laplace_Both_Eval, examples/pure_kifmm_laplace_dipoles.py:31-40),
// times 2 pi
__device__ __forceinline__ double dipole_at(double dx, double dy, double ax, double ay) {
  return fma(dx, ax, dy * ay) / fma(ax, ax, ay * ay);
}

template <int R, int NV>
using PairAcc = double[R][NV];

// Potential sums of a table functor: every charge q is staged times KF::kFold,
// so a pair adds q * raw.  Batches of U sources and R targets test their
// arguments together: one pair outside the table path (a coincident pair,
// as a rule) sends its batch to the pair-by-pair path.  Which targets share a
// batch is chance where they stand in no particular order, so a pair's
// arithmetic is its own: both paths add a pair inside the table by the same
// operations, all written out (fma, __dmul_rn), none left to the compiler to
// contract.  Sources alternate between two chains per target (v[r][0], v[r][1])
// by their place in the thread's sequence, whatever U is.
template <class KF, int R, int U, bool DIP, bool CAT>
__device__ __forceinline__ void pot_batch(const KF &K, const double2 *xy, const double *q,
                                          const double2 *dv, const long long *cat,
                                          const double (&x)[R], const double (&y)[R],
                                          const long long (&tc)[R], int j, int G, int check,
                                          double (&v)[R][2]) {
  double s[R][U];
  double ax[DIP ? R : 1][U], ay[DIP ? R : 1][U];
  constexpr unsigned LIMIT = DIP && RCP_RARE < KF::kRare ? RCP_RARE : KF::kRare;
  // a pair inside the table: s its argument, w its charge, (dx, dy) its offset
  auto table_pair = [&](double s, double w, double dx, double dy, int jj, double &o) {
    o = fma(K.at(s), w, o);
    if constexpr (DIP) {
      const double2 d = dv[jj];
      o = fma(fma(d.x, dx, d.y * dy) * INV_2PI, rcp_newton(s), o);
    }
  };
  unsigned key = 0;
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const double2 p = xy[j + i * G];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double dx = x[r] - p.x, dy = y[r] - p.y;
      s[r][i] = K.arg(fma(dy, dy, dx * dx));
      key = max(key, log2_rare_key(s[r][i]));
      if constexpr (DIP) {
        ax[r][i] = dx;
        ay[r][i] = dy;
      }
    }
  }
  if (key < LIMIT) {
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const double c = q[j + i * G];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double w = c;
        if constexpr (CAT) w = cat[j + i * G] == tc[r] ? 0.0 : c;
        table_pair(s[r][i], w, DIP ? ax[DIP ? r : 0][i] : 0.0, DIP ? ay[DIP ? r : 0][i] : 0.0,
                   j + i * G, v[r][i & 1]);
      }
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < U; ++i) {
      const double2 p = xy[j + i * G];
      const double c = q[j + i * G];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double dx = x[r] - p.x, dy = y[r] - p.y;
        const double t = K.arg(fma(dy, dy, dx * dx));
        if constexpr (CAT)
          if (cat[j + i * G] == tc[r]) continue;
        double o = i & 1 ? v[r][1] : v[r][0];
        if (log2_rare_key(t) < LIMIT) {
          table_pair(t, c, dx, dy, j + i * G, o);
        } else if (!(check && dx == 0.0 && dy == 0.0)) {
          // (a coincident pair is skipped when check is set, helpers.py:99-107)
          o = fma(DIP ? K.raw(dx, dy) : K.raw_rare(dx, dy), c, o);
          if constexpr (DIP) {
            const double2 d = dv[j + i * G];
            o = fma(dipole_at(d.x, d.y, dx, dy), INV_2PI, o);
          }
        }
        if (i & 1)
          v[r][1] = o;
        else
          v[r][0] = o;
      }
    }
  }
}

// one pair of a functor without a table form, added to v
template <class KF>
__device__ __forceinline__ double pair_value(const KF &K, double2 p, double x, double y, double q,
                                             int check) {
  const double v = __dmul_rn(K(p.x, p.y, x, y), q);
  return (check && x - p.x == 0.0 && y - p.y == 0.0) ? 0.0 : v;
}

// v[r] += sources lo, lo + G, ... below hi at the targets (x[r], y[r])
template <class KF, int R, bool DIP, bool CAT>
__device__ __forceinline__ void pot_sweep(const KF &K, const double2 *xy, const double *q,
                                          const double2 *dv, const long long *cat,
                                          const double (&x)[R], const double (&y)[R],
                                          const long long (&tc)[R], int lo, int hi, int G,
                                          int check, double (&v)[R][2]) {
  int j = lo;
  if constexpr (KF::kLogTable) {
    constexpr int U = R == 1 ? 4 : 2;
    for (; j + (U - 1) * G < hi; j += U * G)
      pot_batch<KF, R, U, DIP, CAT>(K, xy, q, dv, cat, x, y, tc, j, G, check, v);
    if (U > 2 && j + G < hi) {
      pot_batch<KF, R, 2, DIP, CAT>(K, xy, q, dv, cat, x, y, tc, j, G, check, v);
      j += 2 * G;
    }
    if (j < hi) pot_batch<KF, R, 1, DIP, CAT>(K, xy, q, dv, cat, x, y, tc, j, G, check, v);
  } else {
    for (int c = 0; j < hi; j += G, c ^= 1) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double a = pair_value(K, xy[j], x[r], y[r], q[j], check);
        if constexpr (CAT) a = cat[j] == tc[r] ? 0.0 : a;
        if (c)
          v[r][1] += a;
        else
          v[r][0] += a;
      }
    }
  }
}

// v[r] = (u, gx, gy) sums of potential and target gradient; table functors
// sum raw values (factors kFold, grad_fold applied at the end)
template <class KF, int R>
__device__ __forceinline__ void grad_sweep(const KF &K, const double2 *xy, const double *q,
                                           const double (&x)[R], const double (&y)[R], int lo,
                                           int hi, int G, int check, double (&v)[R][3]) {
  for (int j = lo; j < hi; j += G) {
    const double2 p = xy[j];
    const double c = q[j];
    if constexpr (KF::kLogTable) {
      // (the targets test together for the common case, each decides for itself)
      constexpr unsigned LIMIT = RCP_RARE < KF::kRare ? RCP_RARE : KF::kRare;
      double dx[R], dy[R], s[R];
      unsigned key[R], most = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        dx[r] = x[r] - p.x;
        dy[r] = y[r] - p.y;
        s[r] = K.arg(fma(dy[r], dy[r], dx[r] * dx[r]));
        key[r] = log2_rare_key(s[r]);
        most = max(most, key[r]);
      }
      auto add = [&](int r, double a, double w) {
        w = __dmul_rn(w, c);
        v[r][0] = fma(a, c, v[r][0]);
        v[r][1] = fma(w, dx[r], v[r][1]);
        v[r][2] = fma(w, dy[r], v[r][2]);
      };
      double a, w;
      if (most < LIMIT) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          K.at_grad(s[r], a, w);
          add(r, a, w);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (key[r] < LIMIT)
            K.at_grad(s[r], a, w);
          else
            K.grad_rare(dx[r], dy[r], check, a, w);
          add(r, a, w);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (!(check && x[r] - p.x == 0.0 && y[r] - p.y == 0.0))
          K.grad(p.x, p.y, x[r], y[r], c, v[r][0], v[r][1], v[r][2]);
    }
  }
}

// The near field of charges (with dipoles: DIP; leaving out a target's own
// category: CAT) and how a target's sums end: a policy's common part.
// NOUT = 1: potential; NOUT = 3: potential and its target gradient.
template <class KF_, int NOUT_, bool DIP, bool CAT>
struct ChargePolicy {
  using KF = KF_;
  using Kernel = KF;
  static constexpr int NOUT = NOUT_, NV = NOUT == 1 ? 2 : 3;
  static constexpr int SMAX = 512;  // sources staged at a time
  static constexpr bool kFolded = KF::kLogTable && NOUT == 1;
  static_assert(!DIP || (KF::kLogTable && NOUT == 1), "dipoles: table Laplace, potential only");
  static_assert(!CAT || (!DIP && NOUT == 1), "categories: potentials of charges only");
  struct Smem {
    double2 xy[SMAX];
    double q[SMAX];
    double2 dv[DIP ? SMAX : 1];
    long long cat[CAT ? SMAX : 1];
    FunctorSmem<KF> f;
  };
  template <int R>
  struct Tgt {
    long long cat[R];
  };
  KernelParams kp;
  const double *sx, *sy, *tau, *dvx, *dvy;
  const int64_t *scat, *tcat;
  int check;
  double *out;
  int64_t ld_out;

  static __device__ __forceinline__ double fold() {
    if constexpr (kFolded)
      return KF::kFold;
    else
      return 1.0;
  }
  template <class S>
  __device__ __forceinline__ KF bind(S &sm) const {
    KF K(kp);
    sm.f.bind(K);
    return K;
  }
  template <class S>
  __device__ __forceinline__ void stage(S &sm, int i, int j) const {
    sm.xy[i] = make_double2(sx[j], sy[j]);
    sm.q[i] = tau[j] * fold();
    if constexpr (DIP) sm.dv[i] = make_double2(dvx[j], dvy[j]);
    if constexpr (CAT) sm.cat[i] = (long long)scat[j];
  }
  __device__ __forceinline__ bool failed() const { return false; }
  template <class T>
  __device__ __forceinline__ void load_target(T &tg, int r, const int *tperm, int t) const {
    if constexpr (CAT) tg.cat[r] = (long long)tcat[tperm[t]];
  }
  template <int R, class S>
  __device__ __forceinline__ void sweep(const KF &K, const S &sm, const double (&x)[R],
                                        const double (&y)[R], const Tgt<R> &tg, int lo, int hi,
                                        int G, double (&v)[R][NV]) const {
    if constexpr (NOUT == 1)
      pot_sweep<KF, R, DIP, CAT>(K, sm.xy, sm.q, sm.dv, sm.cat, x, y, tg.cat, lo, hi, G, check, v);
    else
      grad_sweep<KF, R>(K, sm.xy, sm.q, x, y, lo, hi, G, check, v);
  }
  __device__ __forceinline__ void finish(const double (&v)[NV], double (&o)[NOUT]) const {
    if constexpr (NOUT == 1) {
      o[0] = v[0] + v[1];
    } else if constexpr (KF::kLogTable) {
      o[0] = KF::kFold * v[0];
      o[1] = KF::grad_fold(kp) * v[1];
      o[2] = KF::grad_fold(kp) * v[2];
    } else {
      o[0] = v[0];
      o[1] = v[1];
      o[2] = v[2];
    }
  }
  __device__ __forceinline__ void store(int i, const double (&o)[NOUT]) const {
#pragma unroll
    for (int k = 0; k < NOUT; ++k) out[k * ld_out + i] = o[k];
  }
};

}  // namespace
}  // namespace fmmb
