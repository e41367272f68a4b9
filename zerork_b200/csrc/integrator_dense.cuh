// integrator_dense.cuh -- CTA-per-reactor BDF integration with the Newton
// matrix held as one dense block in shared memory.
//
// The symbolic factorization of the reactor Newton matrix P = I - cJ
// (sparse_lu.h) fills 64-100 % of the dense n x n block for the benchmark
// mechanisms, so the factor is handled as a single dense supernode: P is
// inverted in shared memory by Gauss-Jordan elimination with partial
// pivoting, and every Newton solve is a parallel matrix-vector product.  A
// persistent CTA takes reactors from the work queue; the reactor's BDF state
// (differences, iterate, right-hand sides, weights) and the rate workspace
// live in shared memory, the reactor Jacobian in global memory.  Step
// control is the same as integrator.cu (Shampine-Reichelt BDF with CVODE's
// Newton test and step hysteresis).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "integrator.h"
#include "kinetics_dev.cuh"
#include "reactor_src.cuh"

namespace zrk {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kNewtonMaxIter = 3;
constexpr double kMinFactor = 0.2;
constexpr double kMaxFactor = 10.0;
constexpr double kEtaKeep = 1.5;
constexpr int kMaxl = 10;  // Krylov dimension (no restarts)
constexpr int kPanelMax = 8;  // widest panel of the inversion
constexpr size_t kStateBytes = 1600;  // KernelState
constexpr int kPredBuf = 256;  // widest predictor layer (padded)

struct Smem {
  double *red;  // 128 slots: block sums [0, 16), the right-hand side's [16, 64), change_D [64, 100),
                // Newton norm [100, 116); all of it the inversion's candidates during one
  double *C, *G, *U, *ROP;
  double *D, *y, *f, *f0, *ypred, *psi, *d, *scale, *tmp, *yp;
  void *A;      // n x lda inverse (LT)
  double *rows; // kPanelMax x n pivot rows of the inversion: overlays vectors that are dead then
  double *part; // net_slots partial sums of the net rates: overlays what the reactions leave unread
  int *perm;    // n + 1: low half of entry j the pivot row of column j, high half of entry i
                // the column that row i was the pivot of; entry n the singular flag
  double *wlu;  // n: error-weight scale the stored inverse was formed with
  double *bs;   // n: scaled right-hand side
  double *V;    // FP32 path: (kMaxl + 1) Krylov vectors, then 2 work vectors
  float *mlp;   // learned predictor: two activation buffers of kPredBuf floats
  double *Jsm;  // reactor Jacobian when it is kept in shared memory (spill bit 4)
  const double *ysrc;  // this reactor's mass-fraction sources (global) or null
  ReactorSrc src;      // this reactor's pressure-rate / energy sources and initial state
  // energy-source temperature coupling (global, n each): g = df/dT*,
  // d = dT*/dY, w = (I - c J)^-1 g of the current factor
  double *r1g, *r1d, *r1w;
};

// Doubles of the region that the pivot rows and the predictor share with the
// rates workspace and six vectors.
__host__ __device__ inline size_t dense_rows_doubles(int nsp) {
  const size_t d = 9 * (size_t)nsp + 6;
  return d > kPredBuf ? d : kPredBuf;
}

// What one right-hand-side evaluation used: mixture heat capacity (c_v, or
// c_p for constant pressure), temperature and inverse density.
struct RhsOut {
  double cx, T, v;
};

// Sum over the CTA; every thread gets the same total (deterministic: warp
// trees, then the warps' sums in four chains).  The slots belong to one call
// site: between two uses of them every thread passes another barrier after
// its reads, so one barrier suffices.
__device__ __forceinline__ double block_sum_at(double v, double *slots) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if (lane == 0) slots[threadIdx.x >> 5] = v;
  __syncthreads();
  if (nw == 1) return v;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (i < nw) a[i & 3] += slots[i];
  return (a[0] + a[1]) + (a[2] + a[3]);
}

// The same with slots that any call may have used last.
__device__ __forceinline__ double block_sum(double v, double *red) {
  __syncthreads();
  return block_sum_at(v, red);
}

// Source / constant-pressure adjustment of T and v (reactor_src.cuh).
__device__ __forceinline__ void source_cta(const DevMech &m, const IntegOpts &o, const Smem &s,
                                           double t, const double *y, bool clamp, double v0,
                                           double T_force, double &T, double &v) {
  source_T_v(m, o.cp != 0, s.src, t, y, clamp, o.mmf, v0, T_force, threadIdx.x, blockDim.x,
             [&](double x) { return block_sum(x, s.red); }, T, v);
}

// ydot at y (shared vector) and time t from the start of the call; v0 is the
// reactor's initial inverse density.  Returns 1 if T <= 0 (all threads agree).
// Constant volume: reactor_constant_volume_cpu.cpp:64-128; constant pressure
// (o.cp): reactor_constant_pressure_cpu.cpp:71-135, U then holds h/RT.
// T_force > 0 replaces the energy-source temperature.
__device__ __noinline__ int rhs_cta(const DevMech &m, const IntegOpts &o, const Smem &s,
                                       double v0, double t, const double *y, double *ydot,
                                       bool clamp, RhsOut *out, double T_force = 0.0) {
  const int S = m.nsp, tid = threadIdx.x, nt = blockDim.x;
  const double yS = y[S];
  double T = s.src.fixT ? s.src.T0 : yS * o.Tref;
  if (!(T > 0.0)) return 1;
  if (T > 1.0e4) T = 1.0e4;
  double v = v0;
  if (o.cp || s.src.dpdt != 0.0 || s.src.esrc != 0.0)
    source_cta(m, o, s, t, y, clamp, v0, T_force, T, v);
  // this warp's first block of reactions (3 KB) on its way to L1 during the
  // species pass
  const int lane = tid & 31, w = tid >> 5, nw = nt >> 5;
  auto fetch_block = [&](int b) {
    if (b < m.nblocks && lane < 24)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(m.rxn_slots + (size_t)b * 192 + lane * 8));
  };
  fetch_block(w);
  const double logT = log(T), invT = 1.0 / T;
  const double dens = 1.0 / v;
  const double ush = o.cp ? 0.0 : 1.0;  // h/RT - 1 = u/RT; c_p/R - 1 = c_v/R
  double pc = 0.0, pcv = 0.0;
  for (int k = tid; k < S; k += nt) {
    double ys = y[k];
    if (clamp) ys = clamp_mass_fraction(ys, o.mmf);
    const double c = dens * m.inv_mw[k] * ys;
    s.C[k] = c;
    double cp, h, g;
    nasa_cp_h_g(m.thermo_t + k, T, logT, &cp, &h, &g, S);
    s.G[k] = g;
    s.U[k] = h - ush;
    pc += c;
    pcv += ((cp - ush) * m.ru_inv_mw[k]) * ys;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) pcv += __shfl_xor_sync(kFull, pcv, off);
  if (lane == 0) s.red[32 + w] = pcv;  // read after the barrier of the next sum
  const double Csum = block_sum_at(pc, s.red + 16);
  // blocks of reactions in snake order over the warps
  for (int rr = 0; rr * nw < m.nblocks; ++rr) {
    const int b = rr * nw + ((rr & 1) ? nw - 1 - w : w);
    fetch_block((rr + 1) * nw + ((rr & 1) ? w : nw - 1 - w));
    if (b >= m.nblocks) continue;
    const RxnRec cur = load_slot(m.rxn_slots, b, lane);
    if (!(cur.flags & kNoRxn))
      reaction_item<1, 1>(m, cur, 0, s.C, s.G, s.ROP, &T, &logT, &invT, &Csum, o.lim);
  }
  double cv = 0.0;
  for (int i = 0; i < nw; ++i) cv += s.red[32 + i];
  __syncthreads();
  // Net production rates from equal chunks of the flat list: a chunk's entries
  // and then its rates arrive together, partial sums go to s.part, and a thread
  // a species adds those of its species.  (Eight lanes a species walked lists
  // of very different lengths, some of hundreds of steps, through their
  // pointers: 12.6 K of the
  // right-hand side's 40 K cycles with 160 species.  With few reactions, whose
  // tables L1 holds, that is still the shorter way: 1000 reactors of 27
  // reactions 99 ms, 120 with chunks.)
  double pe = 0.0;
  auto finish = [&](int k, double net) {
    if (s.ysrc) {  // reactor_constant_volume_cpu.cpp:108-113
      const double ys = s.ysrc[k];
      ydot[k] = net * m.mw[k] * v + ys;
      pe += s.U[k] * (net * v + ys * m.inv_mw[k]);
    } else {
      ydot[k] = net * m.mw[k] * v;
      pe += s.U[k] * net * v;
    }
  };
  if (m.net_chunks > 0) {
    const int k0 = min(tid, S - 1), pb = m.net_ptr[k0], pend = m.net_ptr[k0 + 1];
    for (int ch = tid; ch < m.net_chunks; ch += nt) {
      const int4 *ent = m.net_ent + (size_t)(ch >> 5) * m.net_quads * 32 + (ch & 31);
      double *out = s.part + m.net_slot[ch];
      double acc = 0.0;
      for (int q0 = 0; q0 < m.net_quads; q0 += 4) {
        int w[16];
        double r[16];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int4 e = ent[min(q0 + u, m.net_quads - 1) * 32];
          w[4 * u] = e.x;
          w[4 * u + 1] = e.y;
          w[4 * u + 2] = e.z;
          w[4 * u + 3] = e.w;
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) r[u] = s.ROP[w[u] & 0x3fffffff];
#pragma unroll
        for (int u = 0; u < 16; ++u)
          if (q0 + u / 4 < m.net_quads) {
            acc += w[u] < 0 ? -r[u] : r[u];
            if (w[u] & 0x40000000) {
              *out++ = acc;
              acc = 0.0;
            }
          }
      }
    }
    __syncthreads();
    for (int k = tid; k < S; k += nt) {
      const int b = k == tid ? pb : m.net_ptr[k], e = k == tid ? pend : m.net_ptr[k + 1];
      double net = 0.0;
#pragma unroll 4
      for (int i = b; i < e; ++i) net += s.part[i];
      finish(k, net);
    }
  } else {  // few reactions: eight lanes a species, no second barrier
    for (int p0 = tid >> 3; p0 - (lane >> 3) < S; p0 += nt >> 3) {
      const int4 rec = m.sn_rec[min(p0, S - 1)];
      double net = 0.0;
#pragma unroll 4
      for (int e = rec.y + (lane & 7); e < rec.z; e += 8) {
        const int st = m.sn_step[e];
        const double r = s.ROP[st & 0x7fffffff];
        net += st < 0 ? -r : r;
      }
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) net += __shfl_xor_sync(kFull, net, off);
      if (p0 < S && (lane & 7) == 0) finish(rec.x, net);
    }
  }
  const double es = block_sum_at(pe, s.red + 48);
  if (tid == 0)
    ydot[S] = s.src.fixT ? 0.0 : -es * kRuD * yS / cv + (s.src.esrc + s.src.dpdt * v) / (cv * o.Tref);
  if (out) *out = RhsOut{cv, T, v};
  __syncthreads();
  return 0;
}

// Reactor Jacobian (SetupJacobianSparse semantics) into J (global, nnz) at
// y with fy = ydot(t, y).  The concentration derivatives use the reactor's
// inverse density: the initial one at constant volume, the current one at
// constant pressure; the temperature row uses the heat capacities at the
// temperature the right-hand side used.  Under an energy source the
// right-hand side takes T from the energy, T* = T(E0 + esrc t, Y), which
// this Jacobian does not see; the rank-one coupling g d^T (g = df/dT*,
// d_j = dT*/dY_j = -e_j / c_x) goes to s.r1g / s.r1d for the Newton solves.
__device__ __noinline__ int jac_cta(const DevMech &m, const IntegOpts &o, const Smem &s,
                                       double v0, double t, const double *y, const double *fy,
                                       double *J) {
  const int S = m.nsp, n = S + 1, tid = threadIdx.x, nt = blockDim.x;
  int need = 0;
  for (int k = tid; k < S; k += nt) need |= (fabs(y[k]) < o.mmf);
  need = __syncthreads_or(need);
  RhsOut ro;
  if (rhs_cta(m, o, s, v0, t, y, s.tmp, need != 0, &ro)) return 1;
  const double TdC = s.tmp[S];
  const double yS = y[S];
  const double RuTemp = kRuD * yS;
  const double multFact = -1.0 / ro.cx;
  const double T = ro.T, v = o.cp ? ro.v : v0;
  const double ush = o.cp ? 0.0 : 1.0;
  // species columns: a thread a nonzero (the flat item list of devmech.h), as
  // P_ij = dF_i / dC_j; then the temperature row, eight lanes a column
  for (int k = tid; k < S; k += nt) s.yp[k] = m.mw[k] / clamp_mass_fraction(y[k], o.mmf) * v;
  __syncthreads();
#pragma unroll 2
  for (int f = tid; f < m.nj; f += nt) {
    const int2 it = m.jw[f];
    const unsigned short *st = m.jt + m.jt_ptr[f];
    const int j = m.jf_col[f], nd = it.y & 0xffff, nt_ = nd + (it.y >> 16);
    double des = 0.0, cre = 0.0;
    for (int e = 0; e < nt_; ++e) {
      const double r = s.ROP[st[e]];
      if (e < nd) des += r;
      else cre += r;
    }
    const double t2 = s.yp[j];
    J[f + j] = ((0.0 - des * t2) + cre * t2) * (m.mw[it.x] * m.inv_mw[j]);
  }
  __syncthreads();
  for (int j0 = tid >> 3; j0 - ((tid & 31) >> 3) < S; j0 += nt >> 3) {
    const int j = min(j0, S - 1), k1 = m.col_ptr[j + 1] - 1;
    double trow = 0.0;
#pragma unroll 4
    for (int kk = m.col_ptr[j] + (tid & 7); kk < k1; kk += 8) {
      const int row = m.row_idx[kk];
      trow += J[kk] * (m.inv_mw[row] * s.U[row]);
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) trow += __shfl_xor_sync(kFull, trow, off);
    if (j0 < S && (tid & 7) == 0) {
      const double wcol = m.inv_mw[j];
      const double cvj = (nasa_cp(m.thermo + 16 * j, T) - ush) * m.ru_inv_mw[j];
      double tr = trow * m.mw[j] * RuTemp;
      tr += TdC * cvj * m.mw[j];
      tr *= wcol * multFact;
      J[k1] = s.src.fixT ? 0.0 : tr;  // no temperature row when T is not solved
    }
  }
  __syncthreads();
  const double ySp = yS + yS * o.sqrt_ur;
  const double mult = 1.0 / (ySp - yS);
  for (int k = tid; k < S; k += nt) s.yp[k] = y[k];
  if (tid == 0) s.yp[S] = ySp;
  __syncthreads();
  if (rhs_cta(m, o, s, v0, t, s.yp, s.tmp, false, nullptr)) return 1;
  for (int kk = m.col_ptr[S] + tid; kk < m.col_ptr[S + 1]; kk += nt) {
    const int row = m.row_idx[kk];
    J[kk] = (s.tmp[row] - fy[row]) * mult;
  }
  __syncthreads();
  if (s.src.esrc != 0.0) {
    RhsOut r1;
    if (rhs_cta(m, o, s, v0, t, y, s.yp, false, &r1)) return 1;
    for (int j = tid; j < S; j += nt) {
      double cpR, hRT;
      nasa_cp_h(m.thermo + 16 * j, r1.T, &cpR, &hRT);
      s.r1d[j] = -((hRT - ush) * (m.ru_inv_mw[j] * r1.T)) / r1.cx;
    }
    if (tid == 0) s.r1d[S] = 0.0;
    const double Tp = r1.T + r1.T * o.sqrt_ur;
    if (rhs_cta(m, o, s, v0, t, y, s.tmp, false, nullptr, Tp)) return 1;
    for (int i = tid; i < n; i += nt) s.r1g[i] = (s.tmp[i] - s.yp[i]) / (Tp - r1.T);
    __syncthreads();
  }
  return 0;
}

// Newton matrix inverse in shared memory, formed in error-weight-scaled
// coordinates: Pw = W^-1 (I - cJ) W with W = diag(scale), scale = atol +
// rtol |y| of the current step, so entry (i, j) is P_ij scale_j / scale_i,
// the Jacobian of relative changes.  It is far better balanced than P for
// species spanning 20 decades of mass fraction and keeps the inverse
// accurate in the weighted norm the Newton test uses.
//
// Blocked Gauss-Jordan in place with partial pivoting, PB columns at a time
// (Quintana-Orti et al., SIAM J. Sci. Comput. 22 (2001) 1762, with look-ahead
// and without moving rows):
//   * four warps (one, in smaller CTAs) hold the panel of PB columns in
//     registers, a row or two a lane, and exchange its PB pivots with one
//     barrier of their own each; the columns end as W, the panel's part of
//     the inverse;
//   * every other column then changes by one rank-PB product,
//     A_ij = (i a pivot row ? 0 : A_ij) + sum_s W_is R_sj, with R the pivot
//     rows before the update (copied to s.rows);
//   * the next panel's columns are updated first, so the panel's warps factor
//     them while the other warps finish the rest.
// Rows are never swapped: column j's pivot row is noted in perm, unknown j of
// the inverse sits in that row and the right-hand side is gathered in that
// order.  Pivots are the largest by the upper word of |a| (20 mantissa bits,
// ties to the lowest row): one redux instead of a 64-bit shuffle tree.
//
// The sweep by pairs of pivots that this replaces went over the whole matrix
// once per pair (162 passes of shared memory at n = 161) with four block
// barriers each.  Panel width: what the registers of the panel warp hold,
// NC x PB values (128 registers a thread at 512 threads).
//   n = 161 FP64 (160 species)  1,410 K cycles before, 577 K with one panel warp,
//                                434 K with four, the rest in batches of rows on top
//   n = 80 FP64                   407 K cycles before, 172 K, 102 K
template <class LT>
__device__ __forceinline__ unsigned pivot_key(LT a) {
  if constexpr (sizeof(LT) == 8) return (unsigned)__double2hiint(a) & 0x7fffffffu;
  else return __float_as_uint(a) & 0x7fffffffu;
}

// Exchange of the panel columns [k, k + pw) by one warp; `used` has bit r set
// when this lane's row lane + 32 r has been a pivot.  Returns nonzero (all
// lanes) for a singular or non-finite panel.
template <class LT, int NC, int PB>
__device__ __forceinline__ int panel_warp(LT *A, int lda, int n, int k, int pw, int *perm, unsigned &used) {
  constexpr unsigned kInf = sizeof(LT) == 8 ? 0x7ff00000u : 0x7f800000u;
  const int lane = threadIdx.x & 31;
  LT a[NC][PB];
#pragma unroll
  for (int r = 0; r < NC; ++r)
#pragma unroll
    for (int c = 0; c < PB; ++c)
      a[r][c] = (lane + 32 * r < n && c < pw) ? A[(lane + 32 * r) * lda + k + c] : (LT)0;
  // a rolled loop: every exchange rotates the panel left by one column in
  // registers, so the pivot column is always the first
#pragma unroll 1
  for (int t = 0; t < pw; ++t) {
    unsigned key = 0, row = 0xffffffffu;
    bool nan = false;
#pragma unroll
    for (int r = 0; r < NC; ++r) {
      const unsigned q = pivot_key(a[r][0]);
      nan |= q >= kInf;
      if (!(used >> r & 1) && q > key) {  // (rows past n hold zeros)
        key = q;
        row = lane + 32 * r;
      }
    }
    const unsigned best = __reduce_max_sync(kFull, key);
    if (best == 0 || __any_sync(kFull, nan)) return 1;
    const int p = (int)__reduce_min_sync(kFull, key == best ? row : 0xffffffffu);
    const int slot = p >> 5, owner = p & 31;
    LT v[PB];
#pragma unroll
    for (int r = 0; r < NC; ++r)
      if (r == slot)
#pragma unroll
        for (int c = 0; c < PB; ++c) v[c] = a[r][c];
#pragma unroll
    for (int c = 0; c < PB; ++c) v[c] = __shfl_sync(kFull, v[c], owner);
    v[0] = (LT)1 / v[0];
#pragma unroll
    for (int c = 1; c < PB; ++c) v[c] *= v[0];
#pragma unroll
    for (int r = 0; r < NC; ++r) {
      const LT f = a[r][0];
      const bool pr = r == slot && lane == owner;
#pragma unroll
      for (int c = 1; c < PB; ++c) {
        const LT e = a[r][c] - f * v[c];
        a[r][c - 1] = pr ? v[c] : e;
      }
      a[r][PB - 1] = pr ? v[0] : -f * v[0];
    }
    if (lane == owner) used |= 1u << slot;
    if (lane == 0) {
      reinterpret_cast<short *>(perm + k + t)[0] = (short)p;
      reinterpret_cast<short *>(perm + p)[1] = (short)(k + t);
    }
  }
#pragma unroll
  for (int c = 0; c < PB; ++c) {
    const int oc = c + pw - (c + pw >= PB ? PB : 0);  // the column at place c after pw rotations
#pragma unroll
    for (int r = 0; r < NC; ++r)
      if (lane + 32 * r < n && oc < pw) A[(lane + 32 * r) * lda + k + oc] = a[r][c];
  }
  return 0;
}

// The same exchange by warps 0-3 (warp wp the rows 32 wp + lane, and those 128
// further): every warp offers its largest pivot and that row's panel values in
// shared memory (cand: 2 x 4 slots of PB + 1 doubles, used in turn), and one
// barrier of the four warps a pivot settles which one it is.
template <class LT, int RP, int PB>
__device__ __forceinline__ int panel_four(LT *A, int lda, int n, int k, int pw, int *perm, unsigned &used,
                                          double *cand) {
  constexpr unsigned kInf = sizeof(LT) == 8 ? 0x7ff00000u : 0x7f800000u;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, row0 = threadIdx.x;
  LT a[RP][PB];
#pragma unroll
  for (int r = 0; r < RP; ++r)
#pragma unroll
    for (int c = 0; c < PB; ++c)
      a[r][c] = (row0 + 128 * r < n && c < pw) ? A[(row0 + 128 * r) * lda + k + c] : (LT)0;
#pragma unroll 1
  for (int t = 0; t < pw; ++t) {
    unsigned key = 0, row = 0xffffffffu;
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const unsigned q = pivot_key(a[r][0]);
      if ((!(used >> r & 1) || q >= kInf) && q > key) {  // (rows past n hold zeros)
        key = q;
        row = row0 + 128 * r;
      }
    }
    double *slots = cand + (t & 1) * 4 * (PB + 1);
    const unsigned wbest = __reduce_max_sync(kFull, key);
    const unsigned wrow = __reduce_min_sync(kFull, key == wbest ? row : 0xffffffffu);
    if (lane == 0) reinterpret_cast<uint2 *>(slots + wp * (PB + 1) + PB)[0] = make_uint2(wbest, wrow);
#pragma unroll
    for (int r = 0; r < RP; ++r)
      if (row0 + 128 * r == (int)wrow)
#pragma unroll
        for (int c = 0; c < PB; ++c) slots[wp * (PB + 1) + c] = (double)a[r][c];
    asm volatile("bar.sync 1, 128;" ::: "memory");
    unsigned best = 0, p = 0xffffffffu;
    int bw = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // rows of a warp lie between those of others: compare them too
      const uint2 o = reinterpret_cast<const uint2 *>(slots + i * (PB + 1) + PB)[0];
      if (o.x > best || (o.x == best && o.y < p)) {
        best = o.x;
        p = o.y;
        bw = i;
      }
    }
    if (best == 0 || best >= kInf) return 1;  // all four warps alike
    LT v[PB];
#pragma unroll
    for (int c = 0; c < PB; ++c) v[c] = (LT)slots[bw * (PB + 1) + c];
    v[0] = (LT)1 / v[0];
#pragma unroll
    for (int c = 1; c < PB; ++c) v[c] *= v[0];
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const LT f = a[r][0];
      const bool pr = row0 + 128 * r == (int)p;
#pragma unroll
      for (int c = 1; c < PB; ++c) {
        const LT e = a[r][c] - f * v[c];
        a[r][c - 1] = pr ? v[c] : e;
      }
      a[r][PB - 1] = pr ? v[0] : -f * v[0];
      if (pr) {
        used |= 1u << r;
        reinterpret_cast<short *>(perm + k + t)[0] = (short)p;
        reinterpret_cast<short *>(perm + p)[1] = (short)(k + t);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < PB; ++c) {
    const int oc = c + pw - (c + pw >= PB ? PB : 0);  // the column at place c after pw rotations
#pragma unroll
    for (int r = 0; r < RP; ++r)
      if (row0 + 128 * r < n && oc < pw) A[(row0 + 128 * r) * lda + k + oc] = a[r][c];
  }
  return 0;
}

__device__ __forceinline__ int pivot_row(const int *perm, int j) { return perm[j] & 0xffff; }
__device__ __forceinline__ int pivot_col(const int *perm, int i) { return perm[i] >> 16; }

// SH: the matrix and the pivot order are in shared memory.
template <class LT, int NC, int PB, bool SH>
__device__ __noinline__ int invert_cta(const DevMech &m, const Smem &s, const double *J, double c, int n,
                                       int lda) {
  LT *A = (LT *)s.A;
  LT *R = (LT *)s.rows;
  int *perm = s.perm;
  __builtin_assume(__isShared(R));
  if constexpr (SH) {
    __builtin_assume(__isShared(A));
    __builtin_assume(__isShared(perm));
  }
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, w = tid >> 5, nw = nt >> 5;
  for (int i = tid; i < n * lda; i += nt) A[i] = (LT)0;
  for (int i = tid; i < n; i += nt) {
    const double sc = s.scale[i];
    s.wlu[i] = sc;
    s.rows[i] = -c / sc;
    perm[i] = -1;  // no pivot yet: pivot_col < 0
  }
  if (tid == 0) perm[n] = 0;
  __syncthreads();
#pragma unroll 4
  for (int q = tid; q < m.nnz; q += nt) {
    const int rc = m.nz_rc[q], i = rc & 0xffff, j = rc >> 16;
    const double v = s.rows[i] * J[q] * s.wlu[j];
    A[i * lda + j] = (LT)v;
  }
  __syncthreads();
  for (int i = tid; i < n; i += nt) A[i * lda + i] += (LT)1;
  __syncthreads();
  unsigned used = 0;
  const int np = nw >= 4 ? 4 : 1;  // the panel's warps
  auto panel = [&](int k, int pw) {
    if (w >= np) return;
    const int bad = np == 4 ? panel_four<LT, (NC + 3) / 4, PB>(A, lda, n, k, pw, perm, used, s.red)
                            : panel_warp<LT, NC, PB>(A, lda, n, k, pw, perm, used);
    if (bad) perm[n] = 1;
  };
  panel(0, min(PB, n));
  __syncthreads();
  for (int k = 0; k < n && !perm[n]; k += PB) {
    const int pw = min(PB, n - k), k2 = k + pw, pw2 = min(PB, n - k2);
    auto in_panel = [&](int i) { return (unsigned)(pivot_col(perm, i) - k) < (unsigned)pw; };
    for (int q = tid; q < pw * n; q += nt) {  // the pivot rows before the update
      const int t = q / n, j = q - t * n;
      R[q] = A[pivot_row(perm, k + t) * lda + j];
    }
    __syncthreads();
    if (pw2 > 0) {
      for (int q = tid; q < pw2 * n; q += nt) {  // the next panel's columns
        const int t = q / n, i = q - t * n;
        const LT *W = A + i * lda + k;
        LT a = in_panel(i) ? (LT)0 : A[i * lda + k2 + t];
#pragma unroll
        for (int u = 0; u < PB; ++u)
          if (u < pw) a += W[u] * R[u * n + k2 + t];
        A[i * lda + k2 + t] = a;
      }
      __syncthreads();
    }
    const bool ahead = pw2 > 0;
    if (ahead) panel(k2, pw2);
    const bool apart = ahead && nw > np;
    if (!apart || w >= np) {  // the remaining columns, three 32-wide chunks at a time
      const int i0 = apart ? w - np : w, di = apart ? nw - np : nw;
      constexpr int CH = NC < 3 ? NC : 3;
      for (int c0 = 0; c0 < NC; c0 += CH) {
        LT r[PB][CH];
        bool on[CH];
#pragma unroll
        for (int t = 0; t < CH; ++t) {
          const int j = lane + 32 * (c0 + t);
          on[t] = j < n && (j < k || j >= k2 + pw2);
#pragma unroll
          for (int u = 0; u < PB; ++u) r[u][t] = (on[t] && u < pw) ? R[u * n + j] : (LT)0;
        }
        // a batch of rows at a time, every load before the stores (the compiler
        // must keep the order of accesses to A)
        constexpr int RB = sizeof(LT) == 8 && PB * CH >= 24 ? 2 : 3;
        for (int ib = i0; ib < n; ib += RB * di) {
          LT a[RB][CH], wv[RB][PB];
#pragma unroll
          for (int e = 0; e < RB; ++e) {
            const int i = min(ib + e * di, n - 1);
            const LT *row = A + i * lda;
            // (the pivots of the next panel may be noted meanwhile, in entries
            // that this test reads as outside [k, k2))
            const bool piv = in_panel(i);
#pragma unroll
            for (int u = 0; u < PB; ++u) wv[e][u] = u < pw ? row[k + u] : (LT)0;
#pragma unroll
            for (int t = 0; t < CH; ++t) {
              const LT x = on[t] ? row[lane + 32 * (c0 + t)] : (LT)0;
              a[e][t] = piv ? (LT)0 : x;
            }
          }
#pragma unroll
          for (int u = 0; u < PB; ++u)
#pragma unroll
            for (int e = 0; e < RB; ++e)
#pragma unroll
              for (int t = 0; t < CH; ++t) a[e][t] += wv[e][u] * r[u][t];
#pragma unroll
          for (int e = 0; e < RB; ++e)
            if (ib + e * di < n)
#pragma unroll
              for (int t = 0; t < CH; ++t)
                if (on[t]) A[(ib + e * di) * lda + lane + 32 * (c0 + t)] = a[e][t];
        }
      }
    }
    __syncthreads();
  }
  return __syncthreads_or(perm[n]);
}

// Columns of a panel for nc chunks of 32 unknowns.
__host__ __device__ constexpr int panel_width(bool f64, int nc) { return !f64 || nc <= 4 ? 8 : nc <= 6 ? 6 : 4; }

// invert_cta for the register-chunk count nc = ceil(n / 32) (1..8).
template <class LT, bool SH>
__device__ __forceinline__ int invert_any(int nc, const DevMech &m, const Smem &s, const double *J,
                                          double c, int n, int lda) {
  constexpr bool F64 = sizeof(LT) == 8;
  switch (nc) {
    case 1: return invert_cta<LT, 1, 8, SH>(m, s, J, c, n, lda);
    case 2: return invert_cta<LT, 2, 8, SH>(m, s, J, c, n, lda);
    case 3: return invert_cta<LT, 3, 8, SH>(m, s, J, c, n, lda);
    case 4: return invert_cta<LT, 4, 8, SH>(m, s, J, c, n, lda);
    case 5:
    case 6: return invert_cta<LT, 6, panel_width(F64, 6), SH>(m, s, J, c, n, lda);
    default: return invert_cta<LT, 8, panel_width(F64, 8), SH>(m, s, J, c, n, lda);
  }
}

// y = A bs with the stored inverse (rows in pivot order), put(k, y_k) called by
// one thread for each unknown k.  Eight lanes a row, each a contiguous share of
// its columns, and up to three rows a thread that share every right-hand-side
// load; a share of 2 (mod 4) columns and the odd row stride put the lanes of
// two neighbouring rows in different banks.  The caller's barrier precedes it.
template <class LT, class F>
__device__ __forceinline__ void inverse_times_bs(const Smem &s, int n, int lda, F put) {
  const LT *A = (const LT *)s.A;
  const double *bs = s.bs;
  const int *perm = s.perm;
  __builtin_assume(__isShared(A));
  __builtin_assume(__isShared(bs));
  __builtin_assume(__isShared(perm));
  int share = (n + 7) >> 3;
  share += (6 - (share & 3)) & 3;  // the next 2 (mod 4)
  const int g = threadIdx.x & 7, nr = blockDim.x >> 3;
  const int j0 = min(n, g * share), j1 = min(n, j0 + share);
  // every lane of a warp runs the same trips, for the shuffles
  for (int p0 = threadIdx.x >> 3; p0 - ((threadIdx.x & 31) >> 3) < n; p0 += 3 * nr) {
    const int p[3] = {p0, p0 + nr, p0 + 2 * nr};
    double acc[3] = {0.0, 0.0, 0.0};
    const LT *row[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) row[e] = A + min(p[e], n - 1) * lda;
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
      const double v = bs[j];
#pragma unroll
      for (int e = 0; e < 3; ++e) acc[e] += (double)row[e][j] * v;
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
      for (int e = 0; e < 3; ++e) acc[e] += __shfl_xor_sync(kFull, acc[e], o);
#pragma unroll
    for (int e = 0; e < 3; ++e)
      if (g == e && p[e] < n) put(pivot_col(perm, p[e]), acc[e]);
  }
}

// x = (I - c_lu J)^{-1} b with the stored inverse: x = W A (pivot order of
// W^-1 b).
template <class LT>
__device__ void apply_inverse(const Smem &s, int n, int lda, const double *b, double *x) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) s.bs[pivot_col(s.perm, i)] = b[i] / s.wlu[i];
  __syncthreads();
  inverse_times_bs<LT>(s, n, lda, [&](int k, double y) { x[k] = y * s.wlu[k]; });
  __syncthreads();
}

// Energy-source coupling on a Newton solve x = A^-1 b (Sherman-Morrison):
// (A - c g d^T)^-1 b = x + w (r1k d.x) with w = A^-1 g, r1k = c / (1 - c d.w).
__device__ void rank1_fix(const Smem &s, int n, double r1k, double *x) {
  double a = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) a += s.r1d[i] * x[i];
  const double dx = block_sum(a, s.red) * r1k;
  for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] += s.r1w[i] * dx;
  __syncthreads();
}

// (-1)^k binomial(j, k), [k][j]: the difference transform of a unit step
// ratio (Shampine and Reichelt's U).
__device__ const double kSignedBinom[kMaxOrder + 1][kMaxOrder + 1] = {
    {1, 1, 1, 1, 1, 1},   {0, -1, -2, -3, -4, -5}, {0, 0, 1, 3, 6, 10},
    {0, 0, 0, -1, -4, -10}, {0, 0, 0, 0, 1, 5},      {0, 0, 0, 0, 0, -1}};

// Differences of the history for the step size h fac: D <- (R(fac) U)^T D.  A
// thread forms one entry of R U in registers (every thread forming the whole
// product in local arrays took 47 K cycles a call, 2 K now) into mat, 36
// doubles of shared memory.
__device__ void change_D_cta(double *D, int n, int order, double fac, double *mat) {
  constexpr int M = kMaxOrder + 1;
  const double inv[M] = {0.0, 1.0, 0.5, 1.0 / 3.0, 0.25, 0.2};
  __syncthreads();  // mat may still be read, D written
  for (int q = threadIdx.x; q < M * M; q += blockDim.x) {
    const int i = q / M, j = q - i * M;
    double ru = 0.0;
#pragma unroll
    for (int k = 0; k < M; ++k) {
      double r = (k > 0 || i == 0) ? 1.0 : 0.0;
#pragma unroll
      for (int t = 1; t < M; ++t)
        if (k > 0 && t <= i) r *= (t - 1 - fac * k) * inv[t];
      ru += r * kSignedBinom[k][j];
    }
    mat[q] = ru;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    double old[M];
#pragma unroll
    for (int k = 0; k < M; ++k) old[k] = k <= order ? D[k * n + c] : 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      double t = 0.0;
#pragma unroll
      for (int k = 0; k < M; ++k)
        if (k <= order) t += mat[k * M + i] * old[k];
      if (i <= order) D[i * n + c] = t;
    }
  }
  __syncthreads();
}

struct Consts {
  double gam[kMaxOrder + 2], alp[kMaxOrder + 2], econ[kMaxOrder + 2];
};

__host__ __device__ inline void make_consts(Consts &b) {
  const double kap[kMaxOrder + 1] = {0.0, -0.1850, -1.0 / 9.0, -0.0823, -0.0415, 0.0};
  for (int k = 0; k <= kMaxOrder + 1; ++k) {
    double g = 0.0;
    for (int i = 1; i <= k; ++i) g += 1.0 / i;
    b.gam[k] = g;
    const double kk = (k <= kMaxOrder) ? kap[k] : 0.0;
    b.alp[k] = (1.0 - kk) * g;
    b.econ[k] = kk * g + 1.0 / (k + 1);
  }
}


// Left-preconditioned GMRES for (I - cJ) x = b, the Newton system of the
// FP32 path, in the error-weighted coordinates (scale = atol + rtol |y|):
// the operator is applied in FP64 from the stored sparse Jacobian and the
// FP32 inverse is only the preconditioner, so the Newton corrections keep
// FP64 accuracy whatever the single-precision factor loses.  The method is
// SPGMR's (modified Gram-Schmidt, no restarts, x0 = 0, converged when the
// preconditioned residual's weighted 2-norm is <= delta), restated from Saad
// and Schultz, SIAM J. Sci. Stat. Comput. 7 (1986) 856-869; the reference
// plugin drives it through CVODE with PREC_LEFT / MODIFIED_GS
// (applications/cfd_plugin/solver_cvode.cpp:119-141, 201-212).  Every thread
// keeps the same Hessenberg matrix and rotations (the reductions broadcast
// one total), so no thread-0 phase is needed.  Returns 0 when converged, 1
// when the residual was reduced but not below delta, 2 otherwise.
template <class LT>
// Under an energy source the operator and the preconditioner carry the
// rank-one temperature coupling (r1k as in rank1_fix).
__device__ __noinline__ int gmres_cta(const DevMech &m, const Smem &s, const double *J, double c, int n, int lda,
                         double delta, const double *b, double *x, int &iters, double r1k) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const bool r1 = s.src.esrc != 0.0;
  double *V = s.V, *u = s.V + (kMaxl + 1) * n, *z = u + n;
  apply_inverse<LT>(s, n, lda, b, z);
  if (r1) rank1_fix(s, n, r1k, z);
  double a = 0.0;
  for (int i = tid; i < n; i += nt) {
    const double t = z[i] / s.scale[i];
    V[i] = t;
    a += t * t;
  }
  const double beta = sqrt(block_sum(a, s.red));
  if (!isfinite(beta)) return 2;
  if (beta <= delta) {  // the zero initial guess already satisfies the test
    for (int i = tid; i < n; i += nt) x[i] = 0.0;
    __syncthreads();
    return 0;
  }
  double H[kMaxl + 1][kMaxl], cs[kMaxl], sn[kMaxl], g[kMaxl + 1], yk[kMaxl];
  g[0] = beta;
  for (int i = tid; i < n; i += nt) V[i] /= beta;
  int nl = 0;
  double rho = beta;
  bool conv = false;
  for (int l = 0; l < kMaxl; ++l) {
    const double *vl = V + l * n;
    double *w = V + (l + 1) * n;
    double du = 0.0;
    for (int i = tid; i < n; i += nt) {
      u[i] = vl[i] * s.scale[i];
      if (r1) du += s.r1d[i] * u[i];
    }
    if (r1) du = block_sum(du, s.red);
    __syncthreads();
    // (I - cJ) u, eight lanes a row (a thread a row walked some fifty entries
    // on a third of the threads), straight into the inverse's order
    for (int i0 = tid >> 3; i0 - ((tid & 31) >> 3) < n; i0 += nt >> 3) {
      const int i = min(i0, n - 1), q1 = m.jr_ptr[i + 1];
      double jx = 0.0;
#pragma unroll 4
      for (int q = m.jr_ptr[i] + (tid & 7); q < q1; q += 8) jx += J[m.jr_kk[q]] * u[m.jr_col[q]];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) jx += __shfl_xor_sync(kFull, jx, o);
      if (i0 < n && (tid & 7) == 0) {
        if (r1) jx += s.r1g[i] * du;
        s.bs[pivot_col(s.perm, i)] = (u[i] - c * jx) / s.wlu[i];
      }
    }
    __syncthreads();
    if (r1) {
      inverse_times_bs<LT>(s, n, lda, [&](int k, double y) { z[k] = y * s.wlu[k]; });
      __syncthreads();
      rank1_fix(s, n, r1k, z);
      for (int i = tid; i < n; i += nt) w[i] = z[i] / s.scale[i];
    } else {
      inverse_times_bs<LT>(s, n, lda, [&](int k, double y) { w[k] = y * s.wlu[k] / s.scale[k]; });
    }
    __syncthreads();
    for (int k = 0; k <= l; ++k) {  // modified Gram-Schmidt
      const double *vk = V + k * n;
      double d = 0.0;
      for (int i = tid; i < n; i += nt) d += w[i] * vk[i];
      const double h = block_sum(d, s.red);
      H[k][l] = h;
      for (int i = tid; i < n; i += nt) w[i] -= h * vk[i];
    }
    double d2 = 0.0;
    for (int i = tid; i < n; i += nt) d2 += w[i] * w[i];
    const double hn = sqrt(block_sum(d2, s.red));
    for (int k = 0; k < l; ++k) {  // earlier rotations on the new column
      const double h0 = H[k][l], h1 = H[k + 1][l];
      H[k][l] = cs[k] * h0 + sn[k] * h1;
      H[k + 1][l] = -sn[k] * h0 + cs[k] * h1;
    }
    const double a0 = H[l][l];
    double cc, ss;
    if (hn == 0.0) {
      cc = 1.0;
      ss = 0.0;
    } else if (fabs(hn) > fabs(a0)) {
      const double t = a0 / hn;
      ss = 1.0 / sqrt(1.0 + t * t);
      cc = ss * t;
    } else {
      const double t = hn / a0;
      cc = 1.0 / sqrt(1.0 + t * t);
      ss = cc * t;
    }
    H[l][l] = cc * a0 + ss * hn;
    cs[l] = cc;
    sn[l] = ss;
    g[l + 1] = -ss * g[l];
    g[l] = cc * g[l];
    rho = fabs(g[l + 1]);
    nl = l + 1;
    ++iters;
    if (hn > 0.0)
      for (int i = tid; i < n; i += nt) w[i] /= hn;
    if (!isfinite(rho)) return 2;
    if (rho <= delta) {
      conv = true;
      break;
    }
    if (hn == 0.0) break;
  }
  for (int k = nl - 1; k >= 0; --k) {
    double t = g[k];
    for (int j = k + 1; j < nl; ++j) t -= H[k][j] * yk[j];
    yk[k] = t / H[k][k];
  }
  for (int i = tid; i < n; i += nt) {
    double acc = 0.0;
    for (int k = 0; k < nl; ++k) acc += yk[k] * V[k * n + i];
    x[i] = acc * s.scale[i];
  }
  __syncthreads();
  if (conv) return 0;
  return rho < beta ? 1 : 2;
}

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16(x)); }

// Batch-one forward pass of the predictor network (mlp.cu's layers, the
// same BF16 rounding of inputs and hidden activations, FP32 accumulation):
// thread per output, bf16 weights read from global memory (L2-resident).
// Returns the buffer holding the standardised outputs.
__device__ float *mlp_forward_cta(const MlpDev &net, float *a, float *b) {
  for (int l = 0; l < net.layers; ++l) {
    const int K = net.dims[l], N = net.dims[l + 1];
    const __nv_bfloat16 *W = net.w[l];
    const bool hidden = l + 1 < net.layers;
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      float acc = 0.0f;
#pragma unroll 8
      for (int k = 0; k < K; ++k) acc = fmaf(a[k], __bfloat162float(W[(size_t)k * N + j]), acc);
      const float z = acc + net.b[l][j];
      b[j] = hidden ? bf16_round(z / (1.0f + expf(-z))) : z;
    }
    __syncthreads();
    float *t = a;
    a = b;
    b = t;
  }
  return a;
}

// Learned predictor (N3 form): the network's estimate of y(t + h) from the
// last accepted state (row 0 of D) and h replaces the polynomial predictor
// as the Newton starting iterate; ypred, psi and the error estimate keep the
// polynomial predictor, so the error test judges the step exactly as
// without the network.  Inputs: log10 of the clamped mass fractions,
// (T - 1500 K) / 1000 K, log10(P / 1 bar), log10(h); targets: change of
// log10 mass fraction and (T' - T) / 100 K, standardised.
__device__ __noinline__ void predict_cta(const DevMech &m, const IntegOpts &o, const Smem &s, double v, double h) {
  const int S = m.nsp, n = S + 1, tid = threadIdx.x, nt = blockDim.x;
  const PredDev &p = o.pred;
  const double *y0 = s.D;
  double pw = 0.0;
  for (int k = tid; k < S; k += nt) pw += y0[k] * m.inv_mw[k];
  const double iw = block_sum(pw, s.red);
  const double T = y0[S] * o.Tref;
  const double P = kRuD * T * iw / v;
  float *xa = s.mlp, *xb = s.mlp + kPredBuf;
  for (int i = tid; i < p.net.dims[0]; i += nt) {
    double f = 0.0;
    if (i < S) f = log10(fmax(y0[i], 1e-30));
    else if (i == S) f = (T - 1500.0) / 1000.0;
    else if (i == S + 1) f = log10(fmax(P, 1e-300) / 1e5);
    else if (i == S + 2) f = log10(h);
    xa[i] = i < p.net.n_in ? bf16_round((float)((f - p.x_mu[i]) / p.x_sd[i])) : 0.0f;
  }
  __syncthreads();
  const float *r = mlp_forward_cta(p.net, xa, xb);
  for (int i = tid; i < n; i += nt) {
    const double t = (double)r[i] * p.t_sd[i] + p.t_mu[i];
    const double yi = i < S ? exp10(log10(fmax(y0[i], 1e-30)) + t) : (T + 100.0 * t) / o.Tref;
    s.y[i] = yi;
    s.d[i] = yi - s.ypred[i];
  }
  __syncthreads();
}

template <class LT>
__device__ __forceinline__ int attempt_cta(const DevMech &m, const IntegOpts &o, const Consts &bc, const Smem &s,
                           double *J, double v, double t_end, double rtol, double atol,
                           ReactorStats &st, int lda, double &t_done, double t_off, double T_target,
                           double &t_ign, CbCtx &cb) {
  const int n = m.nsp + 1, tid = threadIdx.x, nt = blockDim.x;
  const int nc = (n + 31) / 32;
  auto vrms = [&](const double *x, const double *sc) {
    double a = 0.0;
    for (int i = tid; i < n; i += nt) {
      const double t = x[i] / sc[i];
      a += t * t;
    }
    return sqrt(block_sum(a, s.red) / n);
  };
  double t = 0.0;
  int rc = 0;
  t_done = 0.0;
  double T_prev = s.y[m.nsp] * o.Tref;  // ignition: temperature at the last accepted step
  double r1k = 0.0;  // energy-source coupling of the current factor
  // absolute tolerance of component i: with abstol_dens the species' are
  // abs_tol / molar density (reactor_nvector_serial.cpp:107-119, the
  // correction formed as 1 / (rho / W_k * 1e-3)), at the initial density
  auto atol_of = [&](int i) {
    return (o.abstol_dens && i < m.nsp) ? atol * (1.0 / ((1.0 / v) * m.inv_mw[i] * 1.0e-3)) : atol;
  };
  auto rank1_setup = [&](double cc) {
    if (s.src.esrc == 0.0) return;
    apply_inverse<LT>(s, n, lda, s.r1g, s.r1w);
    double a = 0.0;
    for (int i = tid; i < n; i += nt) a += s.r1d[i] * s.r1w[i];
    const double dw = block_sum(a, s.red);
    r1k = cc / (1.0 - cc * dw);
  };
  st.nrhs++;
  if (rhs_cta(m, o, s, v, t_off, s.y, s.f0, false, nullptr)) return -1;
  for (int i = tid; i < n; i += nt) s.scale[i] = atol_of(i) + fabs(s.y[i]) * rtol;
  __syncthreads();
  const double d0 = vrms(s.y, s.scale), d1 = vrms(s.f0, s.scale);
  double h0 = (d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : 0.01 * d0 / d1;
  if (h0 > t_end) h0 = t_end;
  for (int i = tid; i < n; i += nt) s.tmp[i] = s.y[i] + h0 * s.f0[i];
  __syncthreads();
  double d2 = 0.0;
  st.nrhs++;
  if (rhs_cta(m, o, s, v, t_off + h0, s.tmp, s.f, false, nullptr) == 0) {
    for (int i = tid; i < n; i += nt) s.d[i] = s.f[i] - s.f0[i];
    __syncthreads();
    d2 = vrms(s.d, s.scale) / h0;
  }
  double h1 = (d1 <= 1e-15 && d2 <= 1e-15) ? fmax(1e-6, h0 * 1e-3) : sqrt(0.01 / fmax(d1, d2));
  double h = fmin(100.0 * h0, h1);
  h = fmin(h, o.max_dt);
  h = fmin(h, t_end);
  int q = 1, neq = 0, jac_current = 1, nsteps = 0, pred_fail = 0;
  double c_lu = h / bc.alp[q], crate = 1.0;
  for (int i = tid; i < (kMaxOrder + 3) * n; i += nt) s.D[i] = 0.0;
  __syncthreads();
  for (int i = tid; i < n; i += nt) {
    s.D[i] = s.y[i];
    s.D[n + i] = s.f0[i] * h;
  }
  __syncthreads();
  st.njac++;
  if (jac_cta(m, o, s, v, t_off, s.y, s.f0, J)) { rc = -2; goto failed; }
  st.nlu++;
  if (invert_any<LT, true>(nc, m, s, J, c_lu, n, lda)) { rc = -3; goto failed; }
  rank1_setup(c_lu);
  while (t < t_end) {
    if (nsteps >= o.max_steps) { rc = -4; goto failed; }
    bool accepted = false;
    // the learned predictor starts each step; any rejection falls back to
    // the polynomial predictor for the rest of the step, and after two
    // consecutive failed learned starts the reactor stops consulting the
    // network for the rest of the attempt
    bool use_pred = o.pred.enabled != 0 && pred_fail < 2;
    double safety = 0.9, err_norm = 0.0;
    int nef = 0, ncf = 0;  // this step's error-test and convergence failures
    while (!accepted) {
      if (h > o.max_dt) {
        change_D_cta(s.D, n, q, o.max_dt / h, s.red + 64);
        h = o.max_dt;
      }
      if (t + h > t_end) {
        change_D_cta(s.D, n, q, (t_end - t) / h, s.red + 64);
        h = t_end - t;
      }
      if (!(t + h > t)) { rc = -5; goto failed; }
      const double t_new = t + h;
      for (int i = tid; i < n; i += nt) {
        double a = 0.0, ps = 0.0, dk[kMaxOrder + 1];
#pragma unroll
        for (int k = 0; k <= kMaxOrder; ++k) dk[k] = k <= q ? s.D[k * n + i] : 0.0;  // loads together
#pragma unroll
        for (int k = kMaxOrder; k >= 0; --k)  // the high differences first: they are the smallest
          if (k <= q) {
            a += dk[k];
            if (k > 0) ps += bc.gam[k] * dk[k];
          }
        s.ypred[i] = a;
        s.psi[i] = ps / bc.alp[q];
        s.scale[i] = atol_of(i) + rtol * fabs(a);
        s.y[i] = a;
        s.d[i] = 0.0;
      }
      __syncthreads();
      if (use_pred) predict_cta(m, o, s, v, h);
      const double c = h / bc.alp[q];
      // new factor when c moved by more than 30 % (CVODE's dgmax); a looser
      // rule for the FP32 preconditioner costs more Krylov failures than the
      // factorizations it saves
      if (fabs(c / c_lu - 1.0) > 0.3) {
        st.nlu++;
        c_lu = c;
        crate = 1.0;
        if (invert_any<LT, true>(nc, m, s, J, c, n, lda)) { rc = -3; goto failed; }
        rank1_setup(c);
      }
      const double gscale = (c == c_lu) ? 1.0 : 2.0 / (1.0 + c / c_lu);
      bool conv = false;
      int it;
      double dnorm_old = -1.0;
      for (it = 0; it < kNewtonMaxIter; ++it) {
        st.nrhs++;
        if (rhs_cta(m, o, s, v, t_off + t_new, s.y, s.f, false, nullptr)) break;
        // residual c f - psi - d; on the FP64 path straight into the inverse's
        // order, and the correction goes from the product to the iterate and
        // its norm without a pass of its own
        constexpr bool kDirect = sizeof(LT) == sizeof(double);
        int bad = 0;
        for (int i = tid; i < n; i += nt) {
          const double f = s.f[i], r = c * f - (s.psi[i] + s.d[i]);
          bad |= !isfinite(f);
          s.tmp[i] = r;
          if (kDirect) s.bs[pivot_col(s.perm, i)] = r / s.wlu[i];
        }
        if (__syncthreads_or(bad)) break;
        st.nnewt++;
        double a = 0.0;
        auto correct = [&](int i, double dy) {
          s.y[i] += dy;
          s.d[i] += dy;
          const double tt = dy / s.scale[i];
          a += tt * tt;
        };
        if constexpr (kDirect) {
          if (s.src.esrc == 0.0) {
            inverse_times_bs<LT>(s, n, lda, [&](int k, double y) { correct(k, y * s.wlu[k] * gscale); });
          } else {
            inverse_times_bs<LT>(s, n, lda, [&](int k, double y) { s.yp[k] = y * s.wlu[k]; });
            __syncthreads();
            rank1_fix(s, n, r1k, s.yp);
            for (int i = tid; i < n; i += nt) correct(i, s.yp[i] * gscale);
          }
        } else {
          // Krylov tolerance eps_lin * nlscoef / error constant (WRMS), as a
          // weighted 2-norm.  Unlike CVODE, which accepts a reduced but
          // unconverged residual on the first Newton iteration, every solve
          // must converge: with a single-precision preconditioner a stalled
          // Krylov solve can pass the Newton test with a poor correction,
          // and a failure here costs only a Jacobian update or a step cut.
          const double delta = o.eps_lin * o.nlscoef / bc.econ[q] * sqrt((double)n);
          if (gmres_cta<LT>(m, s, J, c, n, lda, delta, s.tmp, s.yp, st.nkry, r1k) != 0) break;
          // (the Krylov solve uses the current c exactly)
          for (int i = tid; i < n; i += nt) correct(i, s.yp[i]);
        }
        const double dn = sqrt(block_sum_at(a, s.red + 100) / n);
        if (dnorm_old > 0.0) crate = fmax(0.3 * crate, dn / dnorm_old);
        // from a learned starting iterate, convergence is only declared on
        // the last correction itself (two iterations at least): neither the
        // carried rate estimate (the polynomial predictor's start) nor one
        // measured from a large first correction bounds the remaining error
        const double dconv = use_pred ? dn : dn * fmin(1.0, crate);
        if (!(use_pred && it == 0) && bc.econ[q] * dconv <= o.nlscoef) {
          conv = true;
          ++it;
          break;
        }
        if (dnorm_old > 0.0 && dn > 2.0 * dnorm_old) break;
        dnorm_old = dn;
      }
      if (!conv) {
        if (use_pred) {  // the learned start failed: same step from the polynomial predictor
          use_pred = false;
          ++pred_fail;
          continue;
        }
        if (!jac_current) {
          st.nrhs++;
          if (rhs_cta(m, o, s, v, t_off + t_new, s.ypred, s.f0, false, nullptr)) { rc = -6; goto failed; }
          st.njac++;
          if (jac_cta(m, o, s, v, t_off + t_new, s.ypred, s.f0, J)) { rc = -2; goto failed; }
          jac_current = 1;
          st.nlu++;
          c_lu = c;
          crate = 1.0;
          if (invert_any<LT, true>(nc, m, s, J, c, n, lda)) { rc = -3; goto failed; }
          rank1_setup(c);
          continue;
        }
        if (++ncf >= kMaxConvFails) { rc = -8; goto failed; }
        change_D_cta(s.D, n, q, 0.5, s.red + 64);
        h *= 0.5;
        st.nrej++;
        continue;
      }
      safety = 0.9 * (2 * kNewtonMaxIter + 1) / (2.0 * kNewtonMaxIter + it);
      double a = 0.0;
      for (int i = tid; i < n; i += nt) {
        const double e = bc.econ[q] * s.d[i] / s.scale[i];
        a += e * e;
      }
      err_norm = sqrt(block_sum(a, s.red) / n);
      if (!isfinite(err_norm)) { rc = -7; goto failed; }
      if (err_norm > 1.0) {
        if (++nef >= kMaxErrTestFails) { rc = -9; goto failed; }
        use_pred = false;
        st.nrej++;
        if (nef > kErrFailsBeforeCut) {  // order and step cut (integrator.h)
          if (q > 1) {
            --q;
            change_D_cta(s.D, n, q, kEtaMinErrFail, s.red + 64);
          } else {
            st.nrhs++;
            if (rhs_cta(m, o, s, v, t_off + t, s.D, s.tmp, false, nullptr)) { rc = -6; goto failed; }
            for (int i = tid; i < n; i += nt) s.D[n + i] = s.tmp[i] * (h * kEtaMinErrFail);
            __syncthreads();
          }
          h *= kEtaMinErrFail;
          neq = 0;
          continue;
        }
        const double fac = fmax(kMinFactor, safety * pow(err_norm, -1.0 / (q + 1)));
        change_D_cta(s.D, n, q, fac, s.red + 64);
        h *= fac;
        continue;
      }
      if (use_pred) pred_fail = 0;  // the learned start converged and passed
      accepted = true;
      t = t_new;
    }
    ++nsteps;
    st.nsteps++;
    ++neq;
    jac_current = 0;
    const bool keep_prev = T_target > 0.0 && o.stop_ign && t_ign < 0.0;
    for (int i = tid; i < n; i += nt) {
      if (keep_prev) s.tmp[i] = s.D[i];  // the previous accepted state
      const double di = s.d[i];
      double dk[kMaxOrder + 1];
#pragma unroll
      for (int k = 0; k <= kMaxOrder; ++k) dk[k] = k <= q ? s.D[k * n + i] : 0.0;
      s.D[(q + 2) * n + i] = di - s.D[(q + 1) * n + i];
      s.D[(q + 1) * n + i] = di;
      double up = di;
#pragma unroll
      for (int k = kMaxOrder; k >= 0; --k)
        if (k <= q) {
          up += dk[k];
          s.D[k * n + i] = up;
        }
    }
    __syncthreads();
    if (T_target > 0.0) {  // first crossing of T0 + dT_ign, linear between accepted steps
      const double Tn = s.D[n - 1] * o.Tref;
      if (t_ign < 0.0 && Tn >= T_target) {
        const double frac = (Tn > T_prev) ? (T_target - T_prev) / (Tn - T_prev) : 1.0;
        t_ign = t_off + (t - h) + frac * h;
        // the callback's record of CVode's root return (solver_cvode.cpp:249-262)
        const bool cb_end = cb.rec && cb_record(cb, s.D, o.stop_ign ? s.tmp : nullptr, n, q, h,
                                                frac - 1.0, frac, t_ign, s.y, tid, nt);
        if (o.stop_ign || cb_end) {  // stop_after_ignition: the call ends at the crossing
          if (!cb_end)
            for (int i = tid; i < n; i += nt) s.y[i] = s.tmp[i] + frac * (s.D[i] - s.tmp[i]);
          __syncthreads();
          t_done = (t - h) + frac * h;
          return 0;
        }
      }
      T_prev = Tn;
    }
    if (cb.rec && cb_record(cb, s.D, nullptr, n, q, h, 0.0, 0.0, t_off + t, s.y, tid, nt)) {
      __syncthreads();  // the callback asked to stop here
      t_done = t;
      return 0;
    }
    if (neq < q + 1) continue;
    double em = INFINITY, ep = INFINITY;
    {
      double am = 0.0, ap = 0.0;
      for (int i = tid; i < n; i += nt) {
        if (q > 1) {
          const double e = bc.econ[q - 1] * s.D[q * n + i] / s.scale[i];
          am += e * e;
        }
        if (q < kMaxOrder) {
          const double e = bc.econ[q + 1] * s.D[(q + 2) * n + i] / s.scale[i];
          ap += e * e;
        }
      }
      const double sm = block_sum(am, s.red), sp = block_sum(ap, s.red);
      if (q > 1) em = sqrt(sm / n);
      if (q < kMaxOrder) ep = sqrt(sp / n);
    }
    const double fm = (q > 1) ? pow(em, -1.0 / q) : 0.0;
    const double f0 = pow(err_norm, -1.0 / (q + 1));
    const double fp = (q < kMaxOrder) ? pow(ep, -1.0 / (q + 2)) : 0.0;
    int dq = 0;
    double best = f0;
    if (fm > best) { best = fm; dq = -1; }
    if (fp > best) { best = fp; dq = 1; }
    q += dq;
    double fac = fmin(kMaxFactor, safety * best);
    if (fac < kEtaKeep) fac = 1.0;
    change_D_cta(s.D, n, q, fac, s.red + 64);
    h *= fac;
    neq = 0;
  }
  for (int i = tid; i < n; i += nt) s.y[i] = s.D[i];
  __syncthreads();
  t_done = t;
  return 0;
failed:  // D[0] holds the last accepted state (step-size changes keep it)
  for (int i = tid; i < n; i += nt) s.y[i] = s.D[i];
  __syncthreads();
  t_done = t;
  return rc;
}

// spill bits: 1 = rates of progress in a global slice, 2 = BDF differences
// in a global slice (both L2-resident: one slice per resident CTA).
// What the integrator's functions read through references, in shared memory:
// the mechanism's table addresses, options, workspace addresses and method
// constants.  (As kernel parameters and locals they would be copied to the
// stack, which shares what L1 the Newton matrix leaves with the tables; each
// use of a table then waited for its address first, often from L2.)
struct KernelState {
  DevMech m;
  IntegOpts o;
  Smem s;
  Consts bc;
};
static_assert(sizeof(KernelState) <= kStateBytes, "KernelState outgrew its share of shared memory");

template <class LT>
__global__ void __launch_bounds__(512, 1) integrate_dense_kernel(DevMech mp, IntegOpts op, IntegArgs a,
                                                                 int lda, int spill) {
  extern __shared__ double smem_dyn[];
  KernelState &ks = *reinterpret_cast<KernelState *>(smem_dyn);
  const int S = mp.nsp, n = S + 1, N = mp.nstep, tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) {
    ks.m = mp;
    ks.o = op;
    make_consts(ks.bc);
    Smem &s = ks.s;
    double *p = smem_dyn + kStateBytes / sizeof(double);
    double *g = a.rop_scratch + (size_t)blockIdx.x * ((size_t)N + (kMaxOrder + 6) * (size_t)n);
    s.red = p; p += 128;
    // over what is dead then: the inversion's pivot rows (kPanelMax n doubles
    // in the 3 S + 6 n of the rates workspace and six vectors) and the learned
    // predictor's activations
    s.rows = p;
    s.mlp = (float *)p;  // 2 * kPredBuf floats
    double *const end = p + dense_rows_doubles(S);
    s.U = p; p += S;
    s.f = p; p += n;
    s.f0 = p; p += n;
    s.tmp = p; p += n;
    s.yp = p; p += n;
    s.part = p;  // C, G, n doubles and bs: 4 S + 2, dead while the net rates are summed
    s.C = p; p += S;
    s.G = p; p += S;
    p += n;
    s.bs = p;
    p = end;
    if (spill & 1) { s.ROP = g; } else { s.ROP = p; p += N; }
    if (spill & 2) { s.D = g + N; } else { s.D = p; p += (kMaxOrder + 3) * n; }
    s.Jsm = nullptr;
    if (spill & 4) { s.Jsm = p; p += mp.nnz; }
    s.ysrc = nullptr;
    s.r1g = g + N + (kMaxOrder + 3) * n;
    s.r1d = s.r1g + n;
    s.r1w = s.r1d + n;
    s.y = p; p += n;
    s.ypred = p; p += n;
    s.psi = p; p += n;
    s.d = p; p += n;
    s.scale = p; p += n;
    s.wlu = p; p += n;
    s.V = nullptr;
    if (sizeof(LT) == sizeof(float)) {
      s.V = p;
      p += (kMaxl + 3) * n;
    }
    s.perm = (int *)p; p += (n + 1) / 2 + 1;
    s.A = p;
  }
  __syncthreads();
  const DevMech &m = ks.m;
  const IntegOpts &o = ks.o;
  const Smem &s = ks.s;
  const Consts &bc = ks.bc;
  __shared__ int next;
  for (;;) {
    if (tid == 0) next = atomicAdd(a.queue_head, 1);
    __syncthreads();
    const int idx = next;
    __syncthreads();
    if (idx >= a.n_reactors) break;
    const int r = a.order ? a.order[idx] : idx;
    double *J = (spill & 4) ? s.Jsm : a.state + (size_t)r * a.state_stride;
    const double T0 = a.T[r], P0 = a.P[r];
    const double *Y0 = a.Y + (size_t)r * S;
    double pa = 0.0;
    for (int k = tid; k < S; k += nt) pa += Y0[k] * m.inv_mw[k];
    const double mwmix = 1.0 / block_sum(pa, s.red);
    const double v = 1.0 / (P0 * mwmix / (kRuD * T0));
    ReactorSrc src;
    src.dpdt = a.dpdt ? a.dpdt[r] : 0.0;
    src.esrc = a.esrc ? a.esrc[r] : 0.0;
    src.P0 = P0;
    src.ysrc = a.ysrc != nullptr;
    src.fixT = !o.always_T && a.tdel_in && !(a.tdel_in[r] > 0.0);
    src.T0 = T0;
    src.E0 = 0.0;
    if (src.esrc != 0.0 || src.fixT) {  // initial_energy_ (InitializeState)
      double cx;
      mix_energy(m, o.cp != 0, false, T0, Y0, false, 0.0, tid, nt,
                 [&](double x) { return block_sum(x, s.red); }, src.E0, cx);
    }
    if (tid == 0) {  // (the barriers of the sum above end the last reactor's reads)
      ks.s.src = src;
      ks.s.ysrc = a.ysrc ? a.ysrc + (size_t)r * S : nullptr;
    }
    for (int k = tid; k < S; k += nt) s.y[k] = Y0[k];
    if (tid == 0) s.y[S] = T0 / o.Tref;
    __syncthreads();
    ReactorStats rs = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    CbCtx cb{a.cb_rec ? a.cb_rec + (size_t)idx * a.cb_cap * (3 + 2 * (size_t)n) : nullptr, a.cb_cap,
             (a.cb_rec && a.cb_stop) ? a.cb_stop[r] : 0, 0, 0, 0.0};
    double rtol = o.rtol, atol = o.atol;
    int rc = 0;
    // retries (solver_cvode.cpp:227-246): restart the method from the last
    // accepted state for the remaining time with adjusted tolerances;
    // max_steps counts per attempt
    double t_left = a.dt, t_ign = -1.0;
    const double T_target = o.dT_ign > 0.0 ? T0 + o.dT_ign : -1.0;
    for (int attempt = 0;; ++attempt) {
      double t_done = 0.0;
      rc = attempt_cta<LT>(m, o, bc, s, J, v, t_left, rtol, atol, rs, lda, t_done, a.dt - t_left,
                               T_target, t_ign, cb);
      if (rc == 0 || attempt + 1 >= o.max_retries) break;
      cb.ncalls++;  // the failed CVode call counts as a step
      t_left -= t_done;
      rs.retries++;
      atol *= o.retry_atol_factor;
      rtol *= o.retry_rtol_factor;
    }
    rs.status = rc;
    if (rc == 0) {
      double pb = 0.0;
      for (int k = tid; k < S; k += nt) {
        const double ys = s.y[k];
        a.Y[(size_t)r * S + k] = ys;
        pb += ys * m.inv_mw[k];
      }
      const double mw2 = 1.0 / block_sum(pb, s.red);
      const double Tn = end_temperature(m, o.cp != 0, s.src, a.dt, s.y, s.y[S] * o.Tref, tid, nt,
                                        [&](double x) { return block_sum(x, s.red); });
      if (tid == 0) {
        a.T[r] = Tn;
        a.P[r] = end_pressure(o.cp != 0, s.src, a.dt, Tn, mw2, v);
      }
    }
    if (tid == 0) {
      a.v[r] = v;
      if (a.stats) a.stats[r] = rs;
      if (a.cb_cnt) a.cb_cnt[r] = cb.cnt;
      if (a.t_ign) a.t_ign[r] = t_ign;
    }
    __syncthreads();
  }
}


template <class LT>
cudaError_t launch_dense(const DevMech &m, const IntegOpts &o, const IntegArgs &a, int threads,
                         int ctas, int spill, size_t smem, int lda, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(integrate_dense_kernel<LT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // shared memory for the CTAs that can be resident (registers: 512 threads
  // in all), the rest of the SM's 256 KB for L1, which holds the tables
  const size_t want = (smem + 1024) * std::max(1, 512 / std::max(threads, 1));
  const int pct = (int)std::min<size_t>(100, (100 * want + 228 * 1024 - 1) / (228 * 1024));
  e = cudaFuncSetAttribute(integrate_dense_kernel<LT>, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
  if (e != cudaSuccess) return e;
  integrate_dense_kernel<LT><<<ctas, threads, smem, stream>>>(m, o, a, lda, spill);
  return cudaGetLastError();
}

}  // namespace

// One translation unit per factor type (integrator_dense_f64.cu,
// integrator_dense_f32.cu) so the two compile in parallel.
cudaError_t launch_integrate_dense_f64(const DevMech &m, const IntegOpts &o, const IntegArgs &a,
                                       int threads, int ctas, int spill, size_t smem, int lda,
                                       cudaStream_t stream);
cudaError_t launch_integrate_dense_f32(const DevMech &m, const IntegOpts &o, const IntegArgs &a,
                                       int threads, int ctas, int spill, size_t smem, int lda,
                                       cudaStream_t stream);

}  // namespace zrk
