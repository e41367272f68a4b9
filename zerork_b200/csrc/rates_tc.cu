// rates_tc.cu -- rates of progress and species production rates from
// temperature and concentrations, for many states at once: the computation
// behind zerork::mechanism::getReactionRates / getReactionRatesLimiter
// (src/zerork/mechanism.cpp:556-620, perf_net.cpp:126-274) and
// mechanism_cuda::getReactionRates(Limiter)_CUDA_mr_dev
// (src/zerork/mechanism_cuda.h:19-45).
//
// Same tiling as the fused rates + Jacobian kernel (kinetics.cu): a CTA works
// on tiles of TS states, a group of TS / V threads owns one work item
// (species or reaction) for all states of the tile, and states are the fast
// index of every array (x[item * ld + state]).  The temperature is used as
// given (no clamp: the reactor clamps before calling these entry points) and
// the pressure of PLOG reactions is the concentrations' Csum Ru T
// (rate_const.cpp:548-567).
#include <cuda_runtime.h>

#include <cstdint>

#include "devmech.h"
#include "kinetics.h"
#include "kinetics_dev.cuh"

namespace zrk {
namespace {

template <int TS, int V, int MINB>
__global__ void __launch_bounds__(256, MINB) rates_tc_kernel(DevMech m, int n, int ld,
                                                      const double *__restrict__ Tin,
                                                      const double *__restrict__ Cin,
                                                      const double *__restrict__ lim_step,
                                                      double *__restrict__ net,
                                                      double *__restrict__ cre_out,
                                                      double *__restrict__ des_out,
                                                      double *__restrict__ rop_out, int vec) {
  constexpr int GS = TS / V;
  extern __shared__ __align__(16) double smem_dyn[];
  const int S = m.nsp, N = m.nstep;
  const int NW = blockDim.x >> 5, NG = blockDim.x / GS;
  const int g = threadIdx.x / GS, q = threadIdx.x % GS * V, w = threadIdx.x >> 5;
  const bool wlead = (threadIdx.x & 31) < GS;
  double *sC = smem_dyn, *sG = sC + S * TS, *sROP = sG + S * TS, *sPart = sROP + (size_t)N * TS;
#define FORV _Pragma("unroll") for (int k = 0; k < V; ++k)
  const int ntiles = (n + TS - 1) / TS;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int st0 = tile * TS + q;
    bool valid[V];
    FORV valid[k] = st0 + k < n;
    const bool wide = V > 1 && vec && valid[V - 1];  // 16-byte global accesses
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
    double T[V], logT[V], invT[V], Csum[V];
    FORV {
      T[k] = valid[k] ? Tin[st0 + k] : 1000.0;
      logT[k] = log(T[k]);
      invT[k] = 1.0 / T[k];
    }
    // concentrations and g/RT; partial concentration sums per warp
    {
      double pc[V];
      FORV pc[k] = 0.0;
      for (int s = g; s < S; s += NG) {
        const double *th = m.thermo + 16 * s;
        double c[V], gg[V];
        const double *p = Cin + (size_t)s * ld + st0;
        if (wide) ldv<V>(p, c);
        else FORV c[k] = valid[k] ? p[k] : 0.0;
        FORV {
          double cp, h;
          nasa_cp_h_g(th, T[k], logT[k], &cp, &h, &gg[k]);
          pc[k] += c[k];
        }
        stv<V>(sC + s * TS + q, c);
        stv<V>(sG + s * TS + q, gg);
      }
      FORV pc[k] = warp_group_sum<GS>(pc[k]);
      if (wlead) stv<V>(sPart + w * TS + q, pc);
    }
    __syncthreads();
    FORV Csum[k] = 0.0;
    for (int ww = 0; ww < NW; ++ww) {
      double x[V];
      ldv<V>(sPart + ww * TS + q, x);
      FORV Csum[k] += x[k];
    }
    // reactions: both steps of each reaction, the records (sorted by kind and
    // cost) dealt to the groups in snake order (round r gives group g the
    // record at r*NG + g, or r*NG + NG-1-g for odd r) so every group's work is
    // close to the mean; the next one on its way to L1
    for (int rr = 0; rr * NG < m.nrxn; ++rr) {
      const int rp = rr * NG + ((rr & 1) ? NG - 1 - g : g), nx = (rr + 1) * NG + ((rr & 1) ? g : NG - 1 - g);
      if (nx < m.nrxn) asm volatile("prefetch.global.L1 [%0];" ::"l"(m.rxn_by_cost + nx));
      if (rp < m.nrxn)
        reaction_item<TS, V>(m, load_rxn(m.rxn_by_cost + rp), q, sC, sG, sROP, T, logT, invT, Csum, 0.0,
                             lim_step);
    }
    __syncthreads();
    // destruction and creation in ascending step order, net = create - destroy;
    // the longest lists first, in snake order
    for (int rr = 0; rr * NG < S; ++rr) {
      const int sp = rr * NG + ((rr & 1) ? NG - 1 - g : g);
      if (sp >= S) continue;
      const int s = m.spc_order[sp];
      double des[V], cre[V], d[V];
      FORV des[k] = cre[k] = 0.0;
      gather_rop<TS, V>(sROP, m.sd_step, m.sd_ptr[s], m.sd_ptr[s + 1], q, des);
      gather_rop<TS, V>(sROP, m.sc_step, m.sc_ptr[s], m.sc_ptr[s + 1], q, cre);
      FORV d[k] = cre[k] - des[k];
      if (net) put(net + (size_t)s * ld, d);
      if (cre_out) put(cre_out + (size_t)s * ld, cre);
      if (des_out) put(des_out + (size_t)s * ld, des);
    }
    if (rop_out)
      for (int j = g; j < N; j += NG) {
        double r[V];
        ldv<V>(sROP + j * TS + q, r);
        put(rop_out + (size_t)j * ld, r);
      }
    __syncthreads();  // the next tile reuses the workspace
  }
#undef FORV
}

template <int TS, int V, int MINB>
cudaError_t launch_tv(const DevMech &m, const RatesTCArgs &a, int threads, cudaStream_t stream) {
  const int NW = threads / 32;
  const size_t bytes = ((size_t)(2 * m.nsp + m.nstep) * TS + (size_t)NW * TS) * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(rates_tc_kernel<TS, V, MINB>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int ntiles = (a.n + TS - 1) / TS;
  const int grid = ntiles < 8 * sms ? ntiles : 8 * sms;
  const auto al16 = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
  const int vec = a.ld % 2 == 0 && al16(a.C) && al16(a.net) && al16(a.create) && al16(a.destroy) && al16(a.rop);
  rates_tc_kernel<TS, V, MINB><<<grid, threads, bytes, stream>>>(m, a.n, a.ld, a.T, a.C, a.lim_step,
                                                          a.net, a.create, a.destroy, a.rop, vec);
  return cudaGetLastError();
}

}  // namespace

size_t rates_tc_smem_bytes(const DevMech &m, int ts, int threads) {
  return ((size_t)(2 * m.nsp + m.nstep) * ts + (size_t)(threads / 32) * ts) * sizeof(double);
}

cudaError_t launch_rates_tc(const DevMech &m, const RatesTCArgs &a, cudaStream_t stream) {
  if (a.n <= 0) return cudaSuccess;
  // two 8-warp CTAs per SM (16 resident warps, 128 registers each) with 16
  // states per tile where two workspaces fit in shared memory; else one CTA
  // per SM with the largest tile that fits
  const size_t kMax = 227 * 1024, kSm = 228 * 1024;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // up to one state per SM: a CTA a state and a reaction a thread (two rounds
  // of 325 reactions instead of eleven in a 16-state tile of mostly idle lanes)
  if (a.n <= sms && rates_tc_smem_bytes(m, 1, 256) <= kMax) return launch_tv<1, 1, 2>(m, a, 256, stream);
  if (2 * (rates_tc_smem_bytes(m, 16, 256) + 1024) <= kSm) return launch_tv<16, 2, 2>(m, a, 256, stream);
  if (rates_tc_smem_bytes(m, 32, 256) <= kMax) return launch_tv<32, 2, 1>(m, a, 256, stream);
  if (rates_tc_smem_bytes(m, 16, 256) <= kMax) return launch_tv<16, 1, 1>(m, a, 256, stream);
  if (rates_tc_smem_bytes(m, 8, 256) <= kMax) return launch_tv<8, 1, 1>(m, a, 256, stream);
  // a mechanism too large for tiles of 8 runs a state at a time at any size, not
  // only up to one per SM
  if (rates_tc_smem_bytes(m, 1, 256) <= kMax) return launch_tv<1, 1, 2>(m, a, 256, stream);
  return cudaErrorInvalidValue;
}

}  // namespace zrk
