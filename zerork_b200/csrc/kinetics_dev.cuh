// kinetics_dev.cuh -- device helpers shared by the rate and integrator
// kernels: NASA-7 thermo (src/zerork/nasa_poly.cpp:50-172), one reaction's
// two steps (src/zerork/rate_const.cpp:539-582 and perf_net.cpp:190-274),
// and the Jacobian's mass-fraction clamp (reactor_nvector_serial.cpp:629-640).
#pragma once
#include <cuda_runtime.h>

#include "devmech.h"

namespace zrk {

constexpr double kRuD = 8.314462618e3;  // src/zerork/constants.h:10
constexpr double kPatmD = 1.01325e5;    // src/zerork/constants.h:12

constexpr double kLnPatmRu = 2.50033668997960945;  // ln(kPatmD / kRuD)

// Transcendental functions and divisions of K independent arguments side by
// side.  The library's functions and the language's division end in a branch,
// behind which the next call's chain of some twenty dependent operations has
// to wait; here one test covers all K arguments, the chains behind it have no
// branch and interleave, and arguments out of the fast range take the library's
// way.

// Reciprocal of a mid-range number to some 39 bits: the hardware's approximation
// (some 13 bits as measured) and one cubic iteration.  A quotient corrected once by its residual is then
// good to the last place (Markstein, IA-64 and Elementary Functions, 2000).
__device__ __forceinline__ double recip(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ bool mid_range(double x) {
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 523u < 1000u;  // 2^-500 <= |x| < 2^500
}
__device__ __forceinline__ bool not_huge(double x) {
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) < 1523u;  // |x| < 2^500, not NaN
}

// q[i] = a[i] / d[i]: the quotient corrected by its residual (Markstein).  In
// the fast range no quotient overflows (its residual would be infinite and the
// result not a number).
template <int K>
__device__ __forceinline__ void quotients(const double (&a)[K], const double (&d)[K], double (&q)[K]) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < K; ++i) ok = ok && not_huge(a[i]) && mid_range(d[i]);
  if (ok) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const double y = recip(d[i]), g = a[i] * y;
      q[i] = fma(fma(-d[i], g, a[i]), y, g);
    }
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) q[i] = a[i] / d[i];
  }
}

// y[i] = exp(x[i]), fast for |x| < 700: Cody and Waite's reduction by ln 2 in
// two parts (Software Manual for the Elementary Functions, 1980), the Taylor
// polynomial of degree 13 on |r| <= ln 2 / 2 (remainder 4e-18) summed as a
// tree, and the exponent added.  Within an ulp (tests/test_exp_gpu.py).
static __device__ __noinline__ double exp_any(double x) { return exp(x); }

template <int K>
__device__ __forceinline__ void exps(const double (&x)[K], double (&y)[K]) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < K; ++i) ok = ok && (__double2hiint(x[i]) & 0x7fffffff) < 0x4085e000;  // 700
  if (ok) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const double big = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the nearest integer
      const double t = fma(x[i], 1.4426950408889634074, big), k = t - big;
      double r = fma(k, -0.69314718055994530942, x[i]);
      r = fma(k, -2.3190468138462995584e-17, r);  // ln 2 minus its nearest double
      const double r2 = r * r, r4 = r2 * r2, r8 = r4 * r4;
      const double a = fma(1.0 / 6.0, r, 0.5), b = fma(1.0 / 120.0, r, 1.0 / 24.0);
      const double c = fma(1.0 / 5040.0, r, 1.0 / 720.0), d = fma(1.0 / 362880.0, r, 1.0 / 40320.0);
      const double e = fma(1.0 / 39916800.0, r, 1.0 / 3628800.0);
      const double f = fma(1.0 / 6227020800.0, r, 1.0 / 479001600.0);
      const double lo = fma(b, r2, a), mid = fma(d, r2, c), hi = fma(f, r2, e);
      const double p = 1.0 + fma(r2, fma(hi, r8, fma(mid, r4, lo)), r);
      y[i] = __hiloint2double(__double2hiint(p) + (__double2loint(t) << 20), __double2loint(p));
    }
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) y[i] = exp_any(x[i]);
  }
}

// y[i] = ln(x[i]), fast for positive normal numbers: x = 2^k m with m in
// [sqrt(1/2), sqrt 2), ln m = 2 atanh(s) with s = (m - 1) / (m + 1), eleven
// terms of its series (z = s^2 <= 0.0295, remainder 6e-19).
static __device__ __noinline__ double log_any(double x) { return log(x); }

template <int K>
__device__ __forceinline__ void logs(const double (&x)[K], double (&y)[K]) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < K; ++i) ok = ok && (unsigned)(__double2hiint(x[i]) - 0x00100000) < 0x7fe00000u;
  if (ok) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int hi = __double2hiint(x[i]), k = (hi - 0x3fe6a09e) >> 20;  // sqrt(1/2)
      const double m = __hiloint2double(hi - (k << 20), __double2loint(x[i]));
      const double f = m - 1.0, d = m + 1.0, w = recip(d);
      double s = f * w;
      s = fma(fma(-d, s, f), w, s);
      const double z = s * s, z2 = z * z, z4 = z2 * z2, z8 = z4 * z4, s2 = s + s;
      const double p0 = fma(1.0 / 5.0, z, 1.0 / 3.0), p1 = fma(1.0 / 9.0, z, 1.0 / 7.0);
      const double p2 = fma(1.0 / 13.0, z, 1.0 / 11.0), p3 = fma(1.0 / 17.0, z, 1.0 / 15.0);
      const double p4 = fma(1.0 / 21.0, z, 1.0 / 19.0);
      const double p = fma(p4, z8, fma(fma(p3, z2, p2), z4, fma(p1, z2, p0)));
      const double kd = (double)k;
      y[i] = fma(kd, 0.69314718055994530942, s2 + fma(s2 * z, p, kd * 2.3190468138462995584e-17));
    }
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) y[i] = log_any(x[i]);
  }
}

// A mechanism table as the kernel reads it: its copy in the CTA's shared
// memory when the kernel staged the hot tables (tab = the copy of the block
// that starts at the global base), the global table itself for tab = null.
// The staged address is formed from the shared-memory pointer, not by
// offsetting the global one: a pointer derived from a kernel parameter may
// be compiled as a global-space access, which a shared address must not
// reach.  With tab a compile-time null the select folds away.
template <class T>
__device__ __forceinline__ const T *rb(const T *p, const char *tab, const unsigned char *gbase) {
  return tab ? reinterpret_cast<const T *>(
                   tab + (reinterpret_cast<const char *>(p) - reinterpret_cast<const char *>(gbase)))
             : p;
}

// NASA-7 polynomials (src/zerork/nasa_poly.cpp:50-172), one species, one T.
// (ld: distance between a species' coefficients)
__device__ __forceinline__ void nasa_cp_h_g(const double *__restrict__ c, double T, double logT,
                                            double *cp, double *h, double *g, int ld = 1) {
  const double invT = 1.0 / T;
  const double m0 = T * 0.50000000000000000000;
  const double T2 = T * T, T3 = T * T2, T4 = T * T3;
  const double m1 = T2 * 0.33333333333333333333;
  const double m2 = T3 * 0.25000000000000000000;
  const double m3 = T4 * 0.20000000000000000000;
  const double g0 = 1.0 - logT;
  const double g1 = T * -0.50000000000000000000;
  const double g2 = T2 * -0.16666666666666666667;
  const double g3 = T3 * -0.08333333333333333333;
  const double g4 = T4 * -0.05000000000000000000;
  const int o = (T < c[0]) ? 1 : 8;
  const double a1 = c[o * ld], a2 = c[(o + 1) * ld], a3 = c[(o + 2) * ld], a4 = c[(o + 3) * ld],
               a5 = c[(o + 4) * ld], a6 = c[(o + 5) * ld], a7 = c[(o + 6) * ld];
  *cp = a1 + T * (a2 + T * (a3 + T * (a4 + T * a5)));
  *h = a1 + a2 * m0 + a3 * m1 + a4 * m2 + a5 * m3 + a6 * invT;
  *g = a1 * g0 + a2 * g1 + a3 * g2 + a4 * g3 + a5 * g4 + a6 * invT - a7;
}

__device__ __forceinline__ double nasa_cp(const double *__restrict__ c, double T) {
  const int o = (T < c[0]) ? 1 : 8;
  return c[o] + T * (c[o + 1] + T * (c[o + 2] + T * (c[o + 3] + T * c[o + 4])));
}

// A PLOG reaction's forward rate coefficient at (T, P): the Arrhenius lines
// of each distinct pressure summed with the sign of their A, the end
// pressures' values outside [p_min, p_max] and logarithmic interpolation
// between the bracketing pressures inside; zero for T or P <= 0 or a
// non-positive bracketing value (src/zerork/plog_reaction.cpp:166-300,
// without extrapolation as rate_const.cpp:1174-1182 builds them).
__device__ __forceinline__ double plog_at(const DevMech &m, int q, double invT, double logT,
                                          const char *tab = nullptr) {
  const int *lp = rb(m.plog_ln_ptr, tab, m.base);
  const double *sg = rb(m.plog_sgn, tab, m.base), *la = rb(m.plog_lnA, tab, m.base), *ln = rb(m.plog_n, tab, m.base),
               *lt = rb(m.plog_Ta, tab, m.base);
  double k = 0.0;
  for (int l = lp[q]; l < lp[q + 1]; ++l) k += sg[l] * exp(la[l] + logT * ln[l] - invT * lt[l]);
  return k;
}

static __device__ __forceinline__ double plog_rate(const DevMech &m, int j, double T, double invT, double logT,
                                         double P, const char *tab = nullptr) {
  const int *pp = rb(m.plog_pt_ptr, tab, m.base);
  const double *pv = rb(m.plog_p, tab, m.base), *lnp = rb(m.plog_lnp, tab, m.base);
  const int q0 = pp[j], q1 = pp[j + 1];
  if (T <= 0.0 || P <= 0.0) return 0.0;
  if (q1 - q0 == 1 || P <= pv[q0]) return plog_at(m, q0, invT, logT, tab);
  if (P >= pv[q1 - 1]) return plog_at(m, q1 - 1, invT, logT, tab);
  int r = q0;
  while (r + 1 < q1 - 1 && !(pv[r] <= P && P < pv[r + 1])) ++r;
  const double k1 = plog_at(m, r, invT, logT, tab);
  if (k1 <= 0.0) return 0.0;
  const double k2 = plog_at(m, r + 1, invT, logT, tab);
  if (k2 <= 0.0) return 0.0;
  const double e = log(k2 / k1) / (lnp[r + 1] - lnp[r]);
  return k1 * pow(P / pv[r], e);
}

// A reaction record read as six independent 16-byte loads: one memory round
// trip instead of a chain of dependent field loads (generic loads: the
// record may sit in a staged shared-memory copy).
__device__ __forceinline__ RxnRec load_rxn(const RxnRec *p) {
  static_assert(sizeof(RxnRec) == 96, "RxnRec layout");
  const int4 *src = reinterpret_cast<const int4 *>(p);
  int4 b[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) b[i] = src[i];
  RxnRec R;
  memcpy(&R, b, sizeof(R));
  return R;
}

// V consecutive doubles of a workspace row (16-byte aligned for V > 1).
template <int V>
__device__ __forceinline__ void ldv(const double *p, double (&x)[V]) {
  if constexpr (V == 1) {
    x[0] = p[0];
  } else {
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      const double2 t = *reinterpret_cast<const double2 *>(p + k);
      x[k] = t.x;
      x[k + 1] = t.y;
    }
  }
}
template <int V>
__device__ __forceinline__ void stv(double *p, const double (&x)[V]) {
  if constexpr (V == 1) {
    p[0] = x[0];
  } else {
#pragma unroll
    for (int k = 0; k < V; k += 2) *reinterpret_cast<double2 *>(p + k) = make_double2(x[k], x[k + 1]);
  }
}

// Sum over the groups of a warp (lanes q, q+GS, ...) with shuffles; lanes
// q < GS of each warp then hold the warp's partial for their states.
template <int GS>
__device__ __forceinline__ double warp_group_sum(double v) {
#pragma unroll
  for (int o = GS; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Gather-sum of rates of progress over an index list, V states; four rows in
// flight, added in list order.
template <int TS, int V>
__device__ __forceinline__ void gather_rop(const double *__restrict__ sROP, const int *__restrict__ list,
                                           int b, int e, int q, double (&acc)[V]) {
  int i = b;
  for (; i + 3 < e; i += 4) {
    double r[4][V];
#pragma unroll
    for (int u = 0; u < 4; ++u) ldv<V>(sROP + list[i + u] * TS + q, r[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] += r[u][k];
  }
  for (; i < e; ++i) {
    double r[V];
    ldv<V>(sROP + list[i] * TS + q, r);
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] += r[k];
  }
}

// f(row values) for every species of a reaction's side, in order; the rows of
// the first two are read together (PAIR: a latency-bound caller gains, one whose
// warps hide the latency loses the row that a one-species side reads twice:
// 53-species rates from concentrations 1.63 -> 1.54 ms, Jacobians 3.01 -> 3.06).
template <int TS, int V, bool PAIR, class F>
__device__ __forceinline__ void each_row(const double *__restrict__ rows, int q, int count, const short *spc, F f) {
  double a[V], b[V];
  if constexpr (PAIR) {
    ldv<V>(rows + spc[0] * TS + q, a);
    ldv<V>(rows + (count > 1 ? spc[1] : spc[0]) * TS + q, b);
    if (count > 0) f(a);
    if (count > 1) f(b);
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (i < count) {
        ldv<V>(rows + spc[i] * TS + q, a);
        f(a);
      }
  }
  if (count > 2) {
#pragma unroll
    for (int i = 2; i < kMaxSide; ++i)
      if (i < count) {
        ldv<V>(rows + spc[i] * TS + q, a);
        f(a);
      }
  }
}

// Record `lane` of a block of rxn_slots: six coalesced loads a warp.
__device__ __forceinline__ RxnRec load_slot(const int4 *slots, int block, int lane) {
  int4 b[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) b[i] = slots[(block * 6 + i) * 32 + lane];
  RxnRec R;
  memcpy(&R, b, sizeof(R));
  return R;
}

// Third-body concentration: Csum plus the record's efficiency list, four
// entries at a time (the table loads are independent of the sums, which keep
// the list order).
template <int TS, int V>
__device__ __forceinline__ void third_body(const Eff *__restrict__ eff, int ne, int q, const double *__restrict__ sC,
                                           const double *Csum, double *Cm) {
#pragma unroll
  for (int k = 0; k < V; ++k) Cm[k] = Csum[k];
  for (int e = 0; e < ne; e += 4) {
    double a[4], c[4][V];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const Eff f = eff[min(e + i, ne - 1)];
      a[i] = e + i < ne ? f.alpha : 0.0;
      ldv<V>(sC + f.spc * TS + q, c[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (e + i < ne)
#pragma unroll
        for (int k = 0; k < V; ++k) Cm[k] += c[i][k] * a[i];
  }
}

// One reaction (both steps) for the V states a thread owns (states q .. q +
// V - 1 of the tile): rate constants, third body, falloff, step limiter
// (one scalar for all steps, or one per step when lim_step is given) and
// concentration products.  gs: the sum of g/RT over products minus reactants.
// The V states and the forward and reverse sides run side by side.  The
// reduced pressure comes from the difference of the two limits' exponents,
// Pr = exp(a_low - a_high) [M], which needs no division; a falloff reaction's
// five or six exponentials, its two logarithms and its quotients then form one
// chain of a few interleaved groups.  (Troe temperatures such as 1e-30 or 1e15,
// with which files switch a term off or on, put an exponent beyond the fast
// range, and that group's exponentials go the library's way one by one: 7 of the
// dimethyl ether mechanism's 14 Troe reactions.)
template <int TS, int V, bool PAIR = true>
__device__ __forceinline__ void reaction_eval(const DevMech &m, const RxnRec &R, int q,
                                              const double *__restrict__ sC,
                                              const double *gs, double *sROP,
                                              const double *T, const double *logT,
                                              const double *invT,
                                              const double *Csum, double lim,
                                              const double *lim_step = nullptr, const char *tab = nullptr) {
  const bool falloff = (R.flags & kFalloff) != 0;
  double Cm[V];
  if (R.flags & (kThirdBody | kFalloff)) {
    const int fs = falloff ? rb(m.fo_spc, tab, m.base)[R.aux] : -1;
    if (fs >= 0) ldv<V>(sC + fs * TS + q, Cm);
    else third_body<TS, V>(rb(m.eff, tab, m.base) + R.e0, R.ne, q, sC, Csum, Cm);
  }
  // exponents first, then the exponentials together: forward, reverse
  double x[2 * V], kk[2 * V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    x[k] = R.lnA + R.n * logT[k] - R.Ta * invT[k];
    x[V + k] = 0.0;
  }
  if (R.flags & kRevArr) {
#pragma unroll
    for (int k = 0; k < V; ++k) x[V + k] = R.lnA_r + R.n_r * logT[k] - R.Ta_r * invT[k];
  } else if (R.flags & kRevKeq) {
#pragma unroll
    for (int k = 0; k < V; ++k) x[V + k] = gs[k] - R.lnA_r * (kLnPatmRu - logT[k]);
  }
  exps<2 * V>(x, kk);
  double kf[V], kr[V];
#pragma unroll
  for (int k = 0; k < V; ++k) kf[k] = kk[k];
  if (R.flags & kPlog) {  // at the pressure of the concentrations, Csum Ru T (rate_const.cpp:548-567)
#pragma unroll
    for (int k = 0; k < V; ++k) kf[k] = plog_rate(m, R.aux, T[k], invT[k], logT[k], Csum[k] * kRuD * T[k], tab);
  }
  if (R.flags & kRevArr) {
#pragma unroll
    for (int k = 0; k < V; ++k) kr[k] = kk[V + k];
  } else {
    const bool keq = (R.flags & kRevKeq) != 0;
#pragma unroll
    for (int k = 0; k < V; ++k) kr[k] = keq ? kk[V + k] * kf[k] : 0.0;
  }
  if (R.flags & kThirdBody) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      kf[k] *= Cm[k];
      kr[k] *= Cm[k];
    }
  }
  if (falloff) {
    const double *p = rb(m.fo_par, tab, m.base) + 8 * R.aux;
    const int ty = rb(m.fo_type, tab, m.base)[R.aux];
    double Pr[V], fT[V], t[V];
#pragma unroll
    for (int k = 0; k < V; ++k) t[k] = (p[0] + p[1] * logT[k] - p[2] * invT[k]) - x[k];
    exps<V>(t, Pr);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      Pr[k] *= Cm[k];
      if (Pr[k] < 1.0e-300) Pr[k] = 1.0e-300;
      fT[k] = 1.0;
    }
    if (ty == kTroe3 || ty == kTroe4) {
      const double p3 = p[3], p4 = p[4], p5 = p[5], p6 = p[6];  // p4, p5: -1 / T***, -1 / T*, or 0
      double u[3 * V], e[3 * V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        u[k] = T[k] * p4;
        u[V + k] = T[k] * p5;
        u[2 * V + k] = ty == kTroe4 ? -p6 * invT[k] : 0.0;
      }
      exps<3 * V>(u, e);
      double w[2 * V], l[2 * V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        double Fc = 0.0;
        if (p4 != 0.0) Fc += (1.0 - p3) * e[k];
        if (p5 != 0.0) Fc += p3 * e[V + k];
        if (ty == kTroe4) Fc += e[2 * V + k];
        if (Fc < 1.0e-300) Fc = 1.0e-300;
        w[k] = Fc;
        w[V + k] = Pr[k];
      }
      logs<2 * V>(w, l);
      const double ln10 = 2.30258509299404568402, ilog = 0.43429448190325182765;  // log10 = ln / ln 10
      double a[V], d[V], r[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const double lF = l[k] * ilog;
        a[k] = l[V + k] * ilog - (0.4 + 0.67 * lF);
        d[k] = (0.75 - 1.27 * lF) - 0.14 * a[k];
      }
      quotients<V>(a, d, r);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        a[k] = l[k] * ilog;
        d[k] = 1.0 + r[k] * r[k];
      }
      quotients<V>(a, d, r);
#pragma unroll
      for (int k = 0; k < V; ++k) r[k] *= ln10;
      exps<V>(r, fT);
    } else if (ty == kSRI) {
      const double p3 = p[3], p4 = p[4], p5 = p[5], p6 = p[6];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const double lPr = log10(Pr[k]);
        const double xp = 1.0 / (1.0 + lPr * lPr);
        double s = p3 * exp(-p4 * invT[k]);
        if (p5 > 0) s += exp(-T[k] * p5);
        s = pow(s, xp);
        s *= p6;
        fT[k] = s * pow(T[k], p[7]);
      }
    }
    double d[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      t[k] = fT[k] * Pr[k];
      d[k] = 1.0 + Pr[k];
    }
    quotients<V>(t, d, fT);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      kf[k] *= fT[k];
      kr[k] *= fT[k];
    }
  }
  if (lim_step) {  // one limit per step (perf_net.cpp:213-224)
    const double lf = lim_step[R.fwd];
    if (0.0 < lf && lf < 1.0e300) {
#pragma unroll
      for (int k = 0; k < V; ++k) kf[k] *= lf / (lf + kf[k]);
    }
    if (R.rev >= 0) {
      const double lr = lim_step[R.rev];
      if (0.0 < lr && lr < 1.0e300) {
#pragma unroll
        for (int k = 0; k < V; ++k) kr[k] *= lr / (lr + kr[k]);
      }
    }
  } else if (0.0 < lim && lim < 1.0e300) {  // the plugin's step_limiter option
    double num[2 * V], den[2 * V], w[2 * V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      num[k] = num[V + k] = lim;
      den[k] = lim + kf[k];
      den[V + k] = lim + kr[k];
    }
    quotients<2 * V>(num, den, w);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      kf[k] *= w[k];
      kr[k] *= w[V + k];
    }
  }
  each_row<TS, V, PAIR>(sC, q, R.nr, R.r, [&](const double (&c)[V]) {
#pragma unroll
    for (int k = 0; k < V; ++k) kf[k] *= c[k];
  });
  stv<V>(sROP + R.fwd * TS + q, kf);
  if (R.rev >= 0) {
    each_row<TS, V, PAIR>(sC, q, R.np, R.p, [&](const double (&c)[V]) {
#pragma unroll
      for (int k = 0; k < V; ++k) kr[k] *= c[k];
    });
    stv<V>(sROP + R.rev * TS + q, kr);
  }
}

// The sum of the g/RT rows over a reaction's products minus its reactants, for
// a reverse rate from the equilibrium constant (else zero).
template <int TS, int V, bool PAIR = true>
__device__ __forceinline__ void gibbs_from_rows(const RxnRec &R, int q, const double *__restrict__ sG,
                                                double (&gs)[V]) {
#pragma unroll
  for (int k = 0; k < V; ++k) gs[k] = 0.0;
  if (R.flags & kRevKeq) {
    each_row<TS, V, PAIR>(sG, q, R.np, R.p, [&](const double (&g)[V]) {
#pragma unroll
      for (int k = 0; k < V; ++k) gs[k] += g[k];
    });
    each_row<TS, V, PAIR>(sG, q, R.nr, R.r, [&](const double (&g)[V]) {
#pragma unroll
      for (int k = 0; k < V; ++k) gs[k] -= g[k];
    });
  }
}

// The same with the g/RT rows of the species: their sum over products minus
// reactants, then the evaluation.
template <int TS, int V>
__device__ __forceinline__ void reaction_item(const DevMech &m, const RxnRec &R, int q,
                                              const double *__restrict__ sC,
                                              const double *__restrict__ sG, double *sROP,
                                              const double *T, const double *logT,
                                              const double *invT,
                                              const double *Csum, double lim,
                                              const double *lim_step = nullptr, const char *tab = nullptr) {
  double gs[V];
  gibbs_from_rows<TS, V>(R, q, sG, gs);
  reaction_eval<TS, V>(m, R, q, sC, gs, sROP, T, logT, invT, Csum, lim, lim_step, tab);
}

__device__ __forceinline__ double clamp_mass_fraction(double y, double mmf) {
  if (fabs(y) < mmf) return (y < 0.0) ? -mmf : mmf;
  return y;
}


}  // namespace zrk
