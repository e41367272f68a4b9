// kinetics_kernel.cuh -- fused FP64 net production rates + sparse analytic Jacobian
// for sm_100a.
//
// One CTA works on a tile of TS independent states at a time.  A "group" of
// TS / V consecutive threads owns one work item (species, reaction or Jacobian
// entry) for all TS states of the tile, V neighbouring states a thread, so
// every table read is a broadcast and every state read/write is a coalesced
// row of the species-major (SoA) arrays  x[item * ld + state].  Intermediate
// per-state vectors (concentrations, g/RT, u/RT, rates of progress) live in a
// workspace of rows of TS doubles, in shared memory or (GLOBAL) in a global
// slice per CTA.
//
// What bounds it: the latency of table and workspace loads and the issue of
// the instructions around them, not HBM or the FP64 units (profiles/).  So
//   * the entries of a row a thread owns are neighbours: one 16-byte access;
//   * reactions are sorted by kind and cost and dealt in snake order, so the
//     groups of a warp run the same code; records are fetched one ahead;
//   * the Jacobian's entries carry their first four rate indices in one
//     16-byte record, fetched one ahead, whose four rows are read together;
//   * the rates at the perturbed temperature are not evaluated again: with
//     unchanged concentrations a rate of progress changes by the factor of its
//     rate constant, and the temperature column needs only the changes.
//
// Semantics follow the reference operation for operation:
//   * rate constants   : src/zerork/rate_const.cpp:539-582 (Arrhenius :669-687,
//                        Keq :690-731, third body :862-888, falloff :890-1012)
//   * rates            : src/zerork/perf_net.cpp:190-274 (step limiter, ROP,
//                        destruction/creation in ascending step order)
//   * reactor RHS      : applications/cfd_plugin/reactor_constant_volume_cpu.cpp:64-128
//   * Jacobian values  : applications/cfd_plugin/reactor_nvector_serial.cpp:610-771
//                        (clamped analytic part, temperature row, forward-
//                        difference temperature column, dC->dY conversion).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "devmech.h"
#include "kinetics.h"
#include "kinetics_dev.cuh"

namespace zrk {

struct Layout {
  int rC, rU, rROP, rG, rPart, rStash, rows;
};

// Workspace rows of TS doubles: concentrations, u/RT, rates of progress (N
// rows), g/RT, two buffers of
// per-warp partial sums (NW = warps; PR >= 2 NW rows) and two rows that keep the temperature
// derivative and heat capacity of the clamped state through the Jacobian
// phase.  In that phase the first g/RT row, which follows the rates of
// progress, is the row of zeros that pads the index records, and the rest of
// the g/RT and partial rows hold the per-(group, column) temperature-row
// partials.
__host__ __device__ inline Layout make_layout(int S, int N, int PR) {
  Layout L;
  L.rC = 0;
  L.rU = S;
  L.rROP = 2 * S;
  L.rG = 2 * S + N;
  L.rPart = 3 * S + N;
  L.rStash = L.rPart + PR;
  L.rows = L.rStash + 2;
  return L;
}

namespace {

constexpr double kRu = kRuD;
constexpr double kPatm = kPatmD;

// r over each of a side's concentrations in turn, as r was multiplied: their
// product alone may underflow where the rate does not.  (Out of line: rare.)
static __device__ __noinline__ double over_each(double r, const double *y, int stride, int count, int s01, int s23,
                                                int s45) {
#pragma unroll 1
  for (int i = 0; i < count; ++i) {
    const int s = i < 2 ? s01 : i < 4 ? s23 : s45;
    r /= y[((i & 1) ? s >> 16 : s & 0xffff) * stride];
  }
  return r;
}

// The rates of progress of one reaction at T become their changes to T' =
// T + dT at the same concentrations.  A rate constant k n^T exp(-Ta/T) changes
// by the factor 1 + e, e = expm1(n dlogT - Ta dinvT), an equilibrium constant
// by that of its g/RT changes (dG rows); the step limiter's k L / (k + L)
// makes it e (1 - w) / (1 + w e) with w = k / (k + L), the limited constant
// over L.  |e| is a few 1e-6 (the step is sqrt(eps) T); below 1e-4 what the four
// terms of the exponential's series leave out is e^4 / 120 < 1e-18 relative, and
// of the limiter's (w e)^4 = 1e-16.  Falloff and PLOG rates, and exponents beyond
// 1e-4, are evaluated at T' and the old rates subtracted.  Returns false, with
// the rates as they were, for those.
template <int TS, int V>
__device__ __forceinline__ bool rop_change(const RxnRec &R, int q, const double *__restrict__ sC,
                                           const double *__restrict__ sdG, double *sROP, const double (&dlogT)[V],
                                           const double (&dinvT)[V], double lim) {
  double xf[V], xr[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    xf[k] = R.n * dlogT[k] - R.Ta * dinvT[k];
    xr[k] = 0.0;
  }
  if (R.flags & kRevArr) {
#pragma unroll
    for (int k = 0; k < V; ++k) xr[k] = R.n_r * dlogT[k] - R.Ta_r * dinvT[k];
  } else if (R.flags & kRevKeq) {
    gibbs_from_rows<TS, V, false>(R, q, sdG, xr);
#pragma unroll
    for (int k = 0; k < V; ++k) xr[k] += xf[k] + R.lnA_r * dlogT[k];
  }
  bool small = true;
#pragma unroll
  for (int k = 0; k < V; ++k) small = small && fabs(xf[k]) < 1e-4 && fabs(xr[k]) < 1e-4;
  if ((R.flags & (kPlog | kFalloff)) || !small) return false;
  const bool limited = 0.0 < lim && lim < 1.0e300;
  auto side = [&](int step, int count, const short *spc, const double (&x)[V]) {
    double r[V], c[V], e[V];
    ldv<V>(sROP + step * TS + q, r);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      e[k] = x[k] * (1.0 + x[k] * (0.5 + x[k] * (1.0 / 6.0 + x[k] * (1.0 / 24.0))));
      c[k] = 1.0;
    }
    if (limited) {
      each_row<TS, V, false>(sC, q, count, spc, [&](const double (&y)[V]) {
#pragma unroll
        for (int k = 0; k < V; ++k) c[k] *= y[k];
      });
#pragma unroll
      for (int k = 0; k < V; ++k)
        if (!(fabs(r[k]) <= fabs(c[k]) * (lim * 1e-11))) {  // w < 1e-11 changes no bit of 1 + e
          double x = r[k] / c[k];
          if (!(fabs(c[k]) >= 1.0e-290))
            x = over_each(r[k], sC + q + k, TS, count, spc[0] | spc[1] << 16, spc[2] | spc[3] << 16,
                          spc[4] | spc[5] << 16);
          const double w = x / lim, we = w * e[k];
          e[k] = e[k] * (1.0 - w) * (1.0 - we * (1.0 - we * (1.0 - we)));
        }
    }
#pragma unroll
    for (int k = 0; k < V; ++k) r[k] *= e[k];
    stv<V>(sROP + step * TS + q, r);
  };
  side(R.fwd, R.nr, R.r, xf);
  if (R.rev >= 0) side(R.rev, R.np, R.p, xr);
  return true;
}

// The sum of g/RT over a reaction's products minus its reactants from the
// species' fits at T (where the g/RT rows hold something else).
template <int V>
__device__ __forceinline__ void gibbs_from_fits(const double *thermo, const RxnRec &R, const double *T,
                                                const double *logT, double (&gs)[V]) {
#pragma unroll
  for (int k = 0; k < V; ++k) gs[k] = 0.0;
#pragma unroll 1
  for (int i = 0; i < R.np + R.nr; ++i) {
    const bool prod = i < R.np;
    int sp = 0;
#pragma unroll
    for (int e = 0; e < kMaxSide; ++e) {  // (a register record is not indexed)
      if (prod && e == i) sp = R.p[e];
      if (!prod && e == i - R.np) sp = R.r[e];
    }
    const double *th = thermo + 16 * sp;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      double cp, h, g;
      nasa_cp_h_g(th, T[k], logT[k], &cp, &h, &g);
      gs[k] += prod ? g : -g;
    }
  }
}

// The full evaluation at T' out of line, for the kernel of more than 16 warps:
// inlined beside the rates' own, its 64 registers a thread spilled in both.
template <int TS>
__device__ __noinline__ void eval_aside(const DevMech &m, const RxnRec *rec, int q, const double *sC, const double *sG,
                                        double *sROP, double T, double logT, double invT, double Csum, double lim,
                                        const char *tab, const double *thermo) {
  const RxnRec R = load_rxn(rec);
  const double t[1] = {T}, l[1] = {logT}, i[1] = {invT}, c[1] = {Csum};
  double gs[1] = {0.0};
  if (R.flags & kRevKeq) gibbs_from_fits<1>(thermo, R, t, l, gs);
  reaction_eval<TS, 1, false>(m, R, q, sC, gs, sROP, t, l, i, c, lim, nullptr, tab);
}

// JAC: with the Jacobian when jac is given; without, never (a kernel of its own
// where the Jacobian's code costs rates alone: more than 16 warps, whose 64
// registers spilled, 32,768 53-species rates 438 -> 268 us, and two resident
// CTAs, the mapping of large calls for rates, 100,003 states 766 -> 603).
template <int TS, int V, bool GLOBAL, int MAXT, bool STAGE, int MINB, bool JAC>
__global__ void __launch_bounds__(MAXT, MINB) rates_jac_kernel(
    const __grid_constant__ DevMech m, int n, int ld, const double *__restrict__ Tin, const double *__restrict__ Pin,
    const double *__restrict__ Y, double *__restrict__ wdot, double *__restrict__ jac,
    double *__restrict__ ydot, KinParams kp, double *__restrict__ gscratch, int slice_doubles,
    int stage_bytes, int spc_bytes, int part_rows, int vec) {
  constexpr int GS = TS / V;
  extern __shared__ __align__(16) double smem_dyn[];
  const int S = m.nsp, N = m.nstep;
  const int NW = blockDim.x >> 5;
  const int NG = blockDim.x / GS;
  const int g = threadIdx.x / GS;
  const int q = threadIdx.x % GS * V;  // first state of the tile that this thread owns
  const int w = threadIdx.x >> 5;
  const bool wlead = (threadIdx.x & 31) < GS;  // holds the warp partial
  const Layout L = make_layout(S, N, part_rows);
  double *ws = GLOBAL ? gscratch + (size_t)blockIdx.x * slice_doubles : smem_dyn;
  // STAGE: the mechanism's hot tables (stage_bytes of them) copied into
  // shared memory after the workspace; every table read below goes to the
  // copy (tab) instead of global memory
  const char *tab = nullptr;
  if constexpr (STAGE) {
    int4 *dst = reinterpret_cast<int4 *>(smem_dyn + (GLOBAL ? 0 : (size_t)L.rows * TS));
    const int4 *src = reinterpret_cast<const int4 *>(m.base);
    for (int i = threadIdx.x; i < stage_bytes / 16; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    tab = reinterpret_cast<const char *>(dst);
  }
  // the species tables after the workspace, when they fit: every phase reads
  // them once or more per item, and what L1 the workspace leaves is the lists'
  const char *stab = nullptr;
  if (!STAGE && spc_bytes) {
    int4 *dst = reinterpret_cast<int4 *>(smem_dyn + (GLOBAL ? 0 : (size_t)L.rows * TS));
    const int4 *src = reinterpret_cast<const int4 *>(m.mw);
    for (int i = threadIdx.x; i < spc_bytes / 16; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    stab = reinterpret_cast<const char *>(dst);
  }
#define TB(f) rb(m.f, tab, m.base)
#define SB(f) (STAGE ? TB(f) : rb(m.f, stab, (const unsigned char *)m.mw))
  double *sC = ws + L.rC * TS, *sU = ws + L.rU * TS, *sG = ws + L.rG * TS;
  double *sPart = ws + L.rPart * TS, *sStash = ws + L.rStash * TS;
  double *sROP = ws + L.rROP * TS;
#define PT(a, ww, k) sPart[((a) * NW + (ww)) * TS + q + (k)]
#define FORV _Pragma("unroll") for (int k = 0; k < V; ++k)
  // All reactions in snake order (round r gives group g the record at r*NG + g,
  // or at r*NG + NG-1-g for odd r, so that the costliest spread over the groups
  // and every group's total is close to the mean), the next record on its way
  // to L1 during this one: body(record, its address)
  auto each_reaction = [&](auto body) {
    const RxnRec *recs = TB(rxn_by_cost);
#pragma unroll 1
    for (int r = 0; r * NG < m.nrxn; ++r) {
      const int at = r * NG + ((r & 1) ? NG - 1 - g : g);
      if constexpr (!STAGE) {
        const int nx = (r + 1) * NG + ((r & 1) ? g : NG - 1 - g);
        if (nx < m.nrxn) asm volatile("prefetch.global.L1 [%0];" ::"l"(recs + nx));
      }
      if (at < m.nrxn) body(load_rxn(recs + at), recs + at);
    }
  };
  // the padding row of the Jacobian's records (the g/RT rows are free then)
  auto zero_row = [&]() {
    for (int i = threadIdx.x; i < TS; i += blockDim.x) sROP[(size_t)N * TS + i] = 0.0;
  };
  const int ntiles = (n + TS - 1) / TS;
  const double dummy_y = 1.0 / S;

  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int st0 = tile * TS + q;
    bool valid[V];
    FORV valid[k] = st0 + k < n;
    const bool wide = V > 1 && vec && valid[V - 1];  // 16-byte global accesses
    auto yload = [&](int s, double (&y)[V]) {
      const double *p = Y + (size_t)s * ld + st0;
      if (wide) ldv<V>(p, y);
      else FORV y[k] = valid[k] ? p[k] : dummy_y;
    };
    auto put = [&](double *row, const double (&x)[V]) {
      double *p = row + st0;
      if (wide) {
        if constexpr (V > 1) {
#pragma unroll
          for (int k = 0; k < V; k += 2)
            __stcs(reinterpret_cast<double2 *>(p + k), make_double2(x[k], x[k + 1]));
        }
      } else {
        FORV if (valid[k]) __stcs(p + k, x[k]);
      }
    };
    // the next tile's inputs on their way to L2
    if (const long nt = (long)(tile + gridDim.x) * TS; nt < n) {
      for (int i = threadIdx.x; i < S; i += blockDim.x)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Y + (size_t)i * ld + nt));
      if (threadIdx.x == 0) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Tin + nt));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Pin + nt));
      }
    }
    // ---- mixture molecular weight partials
    {
      double pa[V];
      FORV pa[k] = 0.0;
      for (int s = g; s < S; s += NG) {
        const double iw = SB(inv_mw)[s];
        double y[V];
        yload(s, y);
        FORV pa[k] += y[k] * iw;
      }
      FORV pa[k] = warp_group_sum<GS>(pa[k]);
      if (wlead) FORV PT(0, w, k) = pa[k];
    }
    __syncthreads();
    // every thread reduces the warp partials of its own states (same order
    // everywhere, so the values agree) instead of a barrier-fenced one-group
    // phase
    double v[V], Tr[V], logT[V], Csum[V], yS[V], td[V];
    FORV {
      double sum = 0.0;
      for (int ww = 0; ww < NW; ++ww) sum += PT(0, ww, k);
      const double T = valid[k] ? Tin[st0 + k] : 1000.0;
      const double P = valid[k] ? Pin[st0 + k] : kPatm;
      yS[k] = T / kp.Tref;
      const double mwmix = 1.0 / sum;
      const double rho = P * mwmix / (kRu * T);
      v[k] = 1.0 / rho;
      double t = yS[k] * kp.Tref;
      if (t > 1.0e4) t = 1.0e4;
      Tr[k] = t;
      logT[k] = log(t);
    }
    __syncthreads();  // the species pass reuses the partial rows
    // Up to three passes over species and reactions, one body of code:
    //   0  rates at (T, C): net production rates and right-hand side
    //   1  the changes of the rates of progress to T' (rop_change), in place:
    //      temperature column, the forward difference of the right-hand side
    //   2  rates of the clamped state (reactor_nvector_serial.cpp:629-640),
    //      only if a mass fraction of the tile is clamped
    // The species columns read the rates of progress of pass 2, or of pass 0
    // when there is no clamping, before pass 1 changes them.
    int need = 0, npass = 1;
#pragma unroll 1
    for (int pass = 0; pass < npass; ++pass) {
      const bool p1 = JAC && pass == 1;
      // temperature of the rates: T' in pass 1
      double Tq[V], lq[V], iq[V];
      FORV {
        Tq[k] = Tr[k];
        lq[k] = logT[k];
        if (p1) {
          Tq[k] = (yS[k] + yS[k] * kp.sqrt_ur) * kp.Tref;
          if (Tq[k] > 1.0e4) Tq[k] = 1.0e4;
          lq[k] = log(Tq[k]);
        }
        iq[k] = 1.0 / Tq[k];
      }
      {
        double pc[V], pcv[V];
        FORV pc[k] = pcv[k] = 0.0;
        for (int s = g; s < S; s += NG) {
          const double *th = SB(thermo) + 16 * s;
          const double iw = SB(inv_mw)[s], riw = SB(ru_inv_mw)[s];
          double y[V], c[V], gg[V], u[V];
          yload(s, y);
          FORV {
            if (pass == 0) need |= (fabs(y[k]) < kp.mmf);
            if (pass == 2) y[k] = clamp_mass_fraction(y[k], kp.mmf);
            c[k] = (1.0 / v[k]) * iw * y[k];
            double cp, h;
            nasa_cp_h_g(th, Tq[k], lq[k], &cp, &h, &gg[k]);
            u[k] = h - 1.0;
            pc[k] += c[k];
            pcv[k] += ((cp - 1.0) * riw) * y[k];
          }
          if (p1) {  // the changes of g/RT
            FORV {
              double cp, h, g0;
              nasa_cp_h_g(th, Tr[k], logT[k], &cp, &h, &g0);
              gg[k] -= g0;
            }
          } else {
            stv<V>(sC + s * TS + q, c);
            stv<V>(sU + s * TS + q, u);
          }
          stv<V>(sG + s * TS + q, gg);
        }
        FORV {
          pc[k] = warp_group_sum<GS>(pc[k]);
          pcv[k] = warp_group_sum<GS>(pcv[k]);
        }
        if (wlead) FORV {
          PT(0, w, k) = pc[k];
          PT(1, w, k) = pcv[k];
        }
      }
      if (pass == 0) {
        need = __syncthreads_or(need);
        if (JAC && jac) npass = need ? 3 : 2;
      } else {
        __syncthreads();
      }
      double cv[V];
      FORV {
        double cs = 0.0, c2 = 0.0;
        for (int ww = 0; ww < NW; ++ww) {
          cs += PT(0, ww, k);
          c2 += PT(1, ww, k);
        }
        Csum[k] = cs;
        cv[k] = c2;
      }
      each_reaction([&](const RxnRec &R, const RxnRec *rec) {
        double f0[V], r0[V];
        if (p1) {
          double dl[V], di[V];
          FORV {
            const double z = (Tq[k] - Tr[k]) / Tr[k];  // sqrt(eps), or 0 beyond the temperature clamp
            dl[k] = z * (1.0 - z * (0.5 - z * (1.0 / 3.0)));  // log(1 + z)
            di[k] = -z * iq[k];
          }
          if (rop_change<TS, V>(R, q, sC, sG, sROP, dl, di, kp.lim)) return;
          ldv<V>(sROP + R.fwd * TS + q, f0);
          if (R.rev >= 0) ldv<V>(sROP + R.rev * TS + q, r0);
        }
        if (MAXT > 512 && p1) {
          if constexpr (MAXT > 512)
            eval_aside<TS>(m, rec, q, sC, sG, sROP, Tq[0], lq[0], iq[0], Csum[0], kp.lim, tab, SB(thermo));
        } else {
          double gs[V];
          if (p1 && (R.flags & kRevKeq)) gibbs_from_fits<V>(SB(thermo), R, Tq, lq, gs);
          else gibbs_from_rows<TS, V, false>(R, q, sG, gs);
          reaction_eval<TS, V, false>(m, R, q, sC, gs, sROP, Tq, lq, iq, Csum, kp.lim, nullptr, tab);
        }
        if (p1) {
          double x[V];
          ldv<V>(sROP + R.fwd * TS + q, x);
          FORV x[k] -= f0[k];
          stv<V>(sROP + R.fwd * TS + q, x);
          if (R.rev >= 0) {
            ldv<V>(sROP + R.rev * TS + q, x);
            FORV x[k] -= r0[k];
            stv<V>(sROP + R.rev * TS + q, x);
          }
        }
      });
      __syncthreads();  // also fences the reads of the partial rows above
      // net rates (pass 1: their changes) and the energy partial
      {
        double pe[V];
        FORV pe[k] = 0.0;
        // every species' terms four a record, the next record in flight during
        // this one; the longest lists first, in snake order
        for (int r = 0; r * NG < S; ++r) {
          const int sp = r * NG + ((r & 1) ? NG - 1 - g : g);
          if (sp >= S) continue;
          const int4 rec = TB(sq_rec)[sp];
          const int s = rec.x, nd = rec.w;
          const int2 *steps = TB(sq_step) + rec.z;
          double net[V], u[V], out[V];
          FORV net[k] = 0.0;
          int2 nx = steps[0];
          for (int pos = 0; pos < rec.y; pos += 4) {
            const int2 it = nx;
            nx = *++steps;
            if (!STAGE && (pos & 63) == 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(steps + 16));
            double x[4][V];
            ldv<V>(sROP + (it.x & 0xffff) * TS + q, x[0]);
            ldv<V>(sROP + (int)((unsigned)it.x >> 16) * TS + q, x[1]);
            ldv<V>(sROP + (it.y & 0xffff) * TS + q, x[2]);
            ldv<V>(sROP + (int)((unsigned)it.y >> 16) * TS + q, x[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (pos + e < rec.y) {
                const double sg = pos + e < nd ? -1.0 : 1.0;
                FORV net[k] = fma(sg, x[e][k], net[k]);
              }
          }
          const double mws = SB(mw)[s];
          if (p1) {
            const double *th = SB(thermo) + 16 * s, *wd = wdot + (size_t)s * ld + st0;
            FORV {
              const double mult = 1.0 / ((yS[k] + yS[k] * kp.sqrt_ur) - yS[k]);
              out[k] = net[k] * mws * v[k] * mult;
              net[k] += valid[k] ? wd[k] : 0.0;
              double cp, h, gg;
              nasa_cp_h_g(th, Tq[k], lq[k], &cp, &h, &gg);
              u[k] = h - 1.0;
            }
            put(jac + (size_t)(TB(col_ptr)[S] + s) * ld, out);
          } else {
            ldv<V>(sU + s * TS + q, u);
            if (pass == 0) {
              put(wdot + (size_t)s * ld, net);
              if (ydot) {
                FORV out[k] = net[k] * mws * v[k];
                put(ydot + (size_t)s * ld, out);
              }
            }
          }
          FORV pe[k] += u[k] * net[k] * v[k];
        }
        FORV pe[k] = warp_group_sum<GS>(pe[k]);
        if (wlead) FORV PT(0, w, k) = pe[k];
        if (!p1) zero_row();
      }
      __syncthreads();
      double tdq[V];
      FORV {
        double es = 0.0;
        for (int ww = 0; ww < NW; ++ww) es += PT(0, ww, k);
        const double ys = p1 ? yS[k] + yS[k] * kp.sqrt_ur : yS[k];
        tdq[k] = -es * kRu * ys / cv[k] + 0.0;
        if (pass == 0) td[k] = tdq[k];
      }
      if (g == 0 && pass == 0 && ydot) put(ydot + (size_t)S * ld, tdq);
      if (g == 0 && p1) {
        double d[V];
        FORV d[k] = (tdq[k] - td[k]) * (1.0 / ((yS[k] + yS[k] * kp.sqrt_ur) - yS[k]));
        put(jac + (size_t)(TB(col_ptr)[S] + S) * ld, d);
      }
      __syncthreads();  // the energy partials are read before their rows are reused
      if (!JAC || jac == nullptr || p1 || (pass == 0 && need)) continue;
      // ---- analytic Jacobian: the species-column entries (the flat item list of
      // devmech.h) in equal work shares over the groups, the temperature row of
      // each column from per-(group, column) partial sums kept in the g/RT and
      // partial rows (free in this phase: after the row of zeros, S + NGj - 1
      // <= S + part_rows - 1 slots of TS doubles)
      {
        int NGj = NG < S + 1 ? NG : S + 1;
        if (NGj > part_rows) NGj = part_rows;
        const int total = TB(jcost)[m.nj];
        double *sTP = sG + TS;
        auto group_of = [&](int f) { return (int)(((long long)TB(jcost)[f] * NGj) / total); };
        // the temperature derivative and heat capacity of the (clamped) state
        // wait in partial rows for the temperature-row pass (fewer live registers)
        if (g == 0) {
          stv<V>(sStash + q, tdq);
          stv<V>(sStash + TS + q, cv);
        }
        if (g < NGj) {
          auto first_of = [&](int gg) {  // first item f with group_of(f) >= gg
            const long long thr = (long long)gg * total;
            int lo = 0, hi = m.nj;
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              if ((long long)TB(jcost)[mid] * NGj >= thr) hi = mid;
              else lo = mid + 1;
            }
            return lo;
          };
          const int f0 = first_of(g), f1 = first_of(g + 1);
          if (f0 < m.nj) {
            int j = 0, hi = S;  // the column holding f0: jf_ptr[j] <= f0 < jf_ptr[j+1]
            while (j < hi) {
              const int mid = (j + hi + 1) >> 1;
              if (TB(jf_ptr)[mid] <= f0) j = mid;
              else hi = mid - 1;
            }
            double t2[V], trow[V], wcol = 0.0;
            auto column = [&]() {
              wcol = SB(inv_mw)[j];
              const double mj = SB(mw)[j];
              double y[V];
              yload(j, y);
              FORV {
                t2[k] = mj / clamp_mass_fraction(y[k], kp.mmf) * v[k];
                trow[k] = 0.0;
              }
            };
            FORV trow[k] = 0.0;
            if (f0 < f1) {
              column();
              int jend = TB(jf_ptr)[j + 1];
              const int4 *items = TB(jit);
              int4 nx = items[f0];
              // list records of this and the next items on their way to L1, a
              // line of each ahead
              auto ahead = [&](const void *p) {
                if constexpr (!STAGE) asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
              };
              const int2 *ext = TB(jext);
              ahead(items + min(f0 + 8, m.nj));
              ahead(ext + nx.w);
              for (int f = f0; f < f1; ++f) {
                const int4 it = nx;
                nx = items[f + 1];  // in flight during this item (the list ends in a sentinel)
                if ((f & 7) == 0) ahead(items + min(f + 16, m.nj));
                while (f == jend) {  // column j ends inside this share
                  stv<V>(sTP + (j + g) * TS + q, trow);
                  ++j;
                  jend = TB(jf_ptr)[j + 1];
                  column();
                }
                const int row = it.x & 0xffff, nd = (int)((unsigned)it.x >> 16);
                const double conv = SB(mw)[row] * wcol;
                double r[4][V], u[V], val[V], odd[V];
                auto rows = [&](int a, int b) {
                  ldv<V>(sROP + (a & 0xffff) * TS + q, r[0]);
                  ldv<V>(sROP + (int)((unsigned)a >> 16) * TS + q, r[1]);
                  ldv<V>(sROP + (b & 0xffff) * TS + q, r[2]);
                  ldv<V>(sROP + (int)((unsigned)b >> 16) * TS + q, r[3]);
                };
                rows(it.y, it.z);
                ldv<V>(sU + row * TS + q, u);
                FORV val[k] = odd[k] = 0.0;
                // destruction terms negative; two chains
                auto add = [&](int pos) {
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const double sg = pos + e < nd ? -1.0 : 1.0;
                    FORV {
                      if (e & 1) odd[k] = fma(sg, r[e][k], odd[k]);
                      else val[k] = fma(sg, r[e][k], val[k]);
                    }
                  }
                };
                add(0);
                if (it.w < nx.w) {  // further terms, four a record, the next one in flight
                  int2 more = ext[it.w];
                  for (int c = it.w; c < nx.w; ++c) {
                    const int2 cur = more;
                    more = ext[min(c + 1, nx.w - 1)];
                    if ((c & 15) == 0) ahead(ext + c + 16);
                    rows(cur.x, cur.y);
                    add(4 * (c - it.w + 1));
                  }
                  ahead(ext + nx.w);
                }
                FORV val[k] += odd[k];
                FORV {
                  val[k] *= t2[k];
                  trow[k] += val[k] * u[k];
                  val[k] *= conv;
                }
                put(jac + (size_t)(f + j) * ld, val);
              }
            }
            // (an empty share inside a column: its slot of that column holds a
            // zero partial)
            stv<V>(sTP + (j + g) * TS + q, trow);
          }
        }
        __syncthreads();
        // temperature row of column j: the partials of groups group_of(first
        // item) .. group_of(last item), in group order
        for (int j = g; j < S; j += NG) {
          const int g0 = group_of(TB(jf_ptr)[j]), g1 = group_of(TB(jf_ptr)[j + 1] - 1);
          double tp[V], t[V], sd[V], sc[V];
          FORV tp[k] = 0.0;
#pragma unroll 1
          for (int gg = g0; gg <= g1; ++gg) {
            ldv<V>(sTP + (j + gg) * TS + q, t);
            FORV tp[k] += t[k];
          }
          const double *th = SB(thermo) + 16 * j;
          ldv<V>(sStash + q, sd);
          ldv<V>(sStash + TS + q, sc);
          FORV {
            const double cvj = (nasa_cp(th, Tr[k]) - 1.0) * SB(ru_inv_mw)[j];
            double tr = tp[k] * (kRu * yS[k]);
            tr += sd[k] * cvj * SB(mw)[j];
            tr *= SB(inv_mw)[j] * (-1.0 / sc[k]);
            t[k] = tr;
          }
          put(jac + (size_t)(TB(jf_ptr)[j + 1] + j) * ld, t);
        }
      }
      __syncthreads();
    }
  }
#undef PT
#undef TB
#undef SB
#undef FORV
}

template <int TS, int V, bool GLOBAL, int MAXT, bool STAGE, int MINB>
cudaError_t launch_one(const DevMech &m, const RatesJacArgs &a, const KinParams &kp,
                       const LaunchCfg &cfg, cudaStream_t stream) {
  constexpr bool kOwn = MAXT > 512 || (MINB == 2 && !GLOBAL);  // rates alone have a kernel of their own
  auto *kern = kOwn && !a.jac ? rates_jac_kernel<TS, V, GLOBAL, MAXT, STAGE, MINB, !kOwn>
                              : rates_jac_kernel<TS, V, GLOBAL, MAXT, STAGE, MINB, true>;
  const int threads = std::min(cfg.warps * 32, MAXT);
  const int ntiles = (a.n + TS - 1) / TS;
  if (ntiles == 0) return cudaSuccess;
  const int stage_bytes = STAGE ? m.hot_bytes : 0;
  const size_t smem = rates_jac_smem_bytes(m, cfg), slice = GLOBAL ? rates_jac_ws_bytes(m, cfg) : 0;
  if (smem > 227 * 1024) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148, per_sm = 1, grid = ntiles;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (GLOBAL) {
    if (cfg.grid > 0) grid = std::min(cfg.grid, ntiles);
    if ((size_t)grid * slice > a.scratch_bytes) return cudaErrorInvalidValue;
  }
  // The smallest shared-memory carve-out that holds the workspace (and the
  // tables beside it), so the rest of the SM's 256 KB stays L1.  With more CTAs
  // than SMs: of CTAs of fewer than 8 warps as many as make 8 (ten species,
  // 65,536 states, 8-state tiles by 4 warps: 990 us with one CTA's share, 522
  // with two), and of those with a global workspace, which have the species
  // tables only, as many as registers allow.
  int ctas = MINB;
  if (grid > sms) ctas = std::max(ctas, (GLOBAL && !STAGE ? 16 : 8) * 32 / threads);
  const int pct = (int)((100 * ctas * (smem + 1024) + 228 * 1024 - 1) / (228 * 1024));
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, pct < 100 ? pct : 100);
  if (e != cudaSuccess) return e;
  if (!GLOBAL && ntiles > sms) {
    // persistent CTAs: one copy of the staged tables each, and the next
    // tile's inputs are fetched ahead
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    grid = std::min(ntiles, sms * std::max(1, per_sm));
  }
  const auto al16 = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
  const int vec = V > 1 && a.ld % 2 == 0 && al16(a.Y) && al16(a.wdot) && al16(a.jac) && al16(a.ydot);
  kern<<<grid, threads, smem, stream>>>(m, a.n, a.ld, a.T, a.P, a.Y, a.wdot, a.jac, a.ydot, kp, a.scratch,
                                        (int)(slice / sizeof(double)), stage_bytes,
                                        rates_jac_species_fit(m, cfg) ? m.spc_bytes : 0, rates_jac_part_rows(m, cfg), vec);
  return cudaGetLastError();
}

}  // namespace

// More CTAs than SMs in a launch with a global workspace.
inline bool many_ctas(const RatesJacArgs &a, const LaunchCfg &cfg) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int ntiles = (a.n + cfg.ts - 1) / cfg.ts;
  return (cfg.grid > 0 ? std::min(cfg.grid, ntiles) : ntiles) > sms;
}

// The kernels of one tile size (one translation unit each, to compile side by
// side).  Up to 8 warps may use 255 registers a thread (128 of them, two CTAs
// resident, on request), up to 16 warps 128, 32 warps (one state per thread
// only) 64: the more warps hide latency, the fewer registers hold values in
// flight.  8 warps with 128 registers instead: 32,768 53-species states, 32-state
// tiles, two states a thread 939 -> 1,005 us, four 911 -> 1,125.  With a global
// workspace and more CTAs than SMs, 128: several are resident then (ten species,
// 65,536 states, 16-state tiles 779 -> 533 us; 53 species 1,152 -> 1,306).
// Staged tables and two resident CTAs only with tiles of at most 16 states
// (larger tiles leave no room).
template <int TS, int V, bool GLOBAL>
cudaError_t launch_tvg(const DevMech &m, const RatesJacArgs &a, const KinParams &kp, const LaunchCfg &cfg,
                       cudaStream_t stream) {
  if constexpr (TS <= 16) {
    if (cfg.stage) {
      if (cfg.warps <= 8) return launch_one<TS, V, GLOBAL, 256, true, 1>(m, a, kp, cfg, stream);
      if (cfg.warps <= 16) return launch_one<TS, V, GLOBAL, 512, true, 1>(m, a, kp, cfg, stream);
      if constexpr (V == 1) return launch_one<TS, V, GLOBAL, 1024, true, 1>(m, a, kp, cfg, stream);
      return cudaErrorInvalidValue;
    }
    if (cfg.minb == 2) return launch_one<TS, V, GLOBAL, 256, false, 2>(m, a, kp, cfg, stream);
  }
  if (cfg.stage || cfg.minb != 1) return cudaErrorInvalidValue;
  if (cfg.warps <= (GLOBAL && many_ctas(a, cfg) ? 0 : 8)) return launch_one<TS, V, GLOBAL, 256, false, 1>(m, a, kp, cfg, stream);
  if (cfg.warps <= 16) return launch_one<TS, V, GLOBAL, 512, false, 1>(m, a, kp, cfg, stream);
  if constexpr (V == 1) return launch_one<TS, V, GLOBAL, 1024, false, 1>(m, a, kp, cfg, stream);
  return cudaErrorInvalidValue;
}

template <int TS, int V>
cudaError_t launch_tv(const DevMech &m, const RatesJacArgs &a, const KinParams &kp, const LaunchCfg &cfg,
                      cudaStream_t stream) {
  return cfg.global_ws ? launch_tvg<TS, V, true>(m, a, kp, cfg, stream)
                       : launch_tvg<TS, V, false>(m, a, kp, cfg, stream);
}

template <int TS>
cudaError_t launch_ts(const DevMech &m, const RatesJacArgs &a, const KinParams &kp, const LaunchCfg &cfg,
                      cudaStream_t stream) {
  switch (cfg.v) {
    case 1: return launch_tv<TS, 1>(m, a, kp, cfg, stream);
    case 2: return launch_tv<TS, 2>(m, a, kp, cfg, stream);
    case 4: return launch_tv<TS, 4>(m, a, kp, cfg, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace zrk
