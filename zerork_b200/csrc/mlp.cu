// mlp.cu -- the learned BDF predictor network: a multilayer perceptron with
// SiLU hidden layers, BF16 weights and activations, FP32 accumulation, FP32
// master weights and Adam moments, trained and evaluated by the kernels in
// this file (no library GEMM).
//
// Layouts (row-major, every dimension padded to a multiple of 16):
//   X_l [batch x K_l] bf16 (layer input), W_l [K_l x N_l] bf16, b_l [N_l] f32,
//   Z_l [batch x N_l] f32 (pre-activation, kept for the backward pass).
//
// The networks are small (three layers of 256 at batches of a few thousand:
// 1.8 GFLOP a training step, 1.1 us at the tensor cores' rate), so a step is
// bound by the chain of dependent launches and by the latency inside each,
// not by arithmetic or bandwidth.  Hence:
//   * one tile routine for all products: 64 x 64 outputs by 4 warps (256 CTAs
//     for 4096 x 256), operands through shared memory by a three-stage
//     cp.async pipeline of 32-deep slices, ldmatrix and m16n8k16 products with
//     FP32 accumulators; transposed operands (X^T dZ, dZ W^T) are read in
//     place and transposed by ldmatrix;
//   * bias, SiLU, its derivative and the loss gradient work on the accumulators;
//   * the weight gradients and bias gradients of all layers form one launch
//     after the input gradients.  Each is one sum over the batch rows in order,
//     not a sum of slices, so a training run repeats bit for bit whatever the
//     tiling; 32 x 64 tiles of every layer run side by side (112 of the network
//     below, on 148 SMs) and last as long as one chain of 4096 / 16 products.
//     (Deeper pipelines, 60 KB in flight instead of 24, changed nothing.  Sums
//     of slices of the batch took 1.11 ms where this takes 1.19.)
// 163-256-256-256-161 on a B200: eight training steps at batch 4096, a forward
// pass of 5,001 rows and the copy of the parameters to the host took 15.2 ms
// with a kernel for each elementwise pass, products straight from global
// memory and one block per weight-gradient tile, and take 1.19 ms now.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <random>
#include <stdexcept>
#include <type_traits>
#include <string>
#include <vector>

#include "../../include/zerork_b200.h"
#include "../../include/zerork_b200_predictor.h"
#include "capi_internal.h"
#include "mlp.h"

namespace zrk {
namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// input: f32 [batch x n_in] (row stride n_in) -> bf16 [batch x K0] zero-padded
__global__ void input_to_bf16(int rows, int n_in, int K0, const float *__restrict__ x, bf16 *__restrict__ X) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)rows * K0) return;
  const int r = (int)(i / K0), c = (int)(i - (long)r * K0);
  X[i] = __float2bfloat16(c < n_in ? x[(size_t)r * n_in + c] : 0.0f);
}

constexpr int kBM = 64, kBN = 64, kBK = 32, kStages = 3;
// Elements of an operand tile of R (the output dimension) x BK in either layout;
// rows padded by 16 bytes: ldmatrix without bank conflicts.
constexpr int tile_elems(int R, int BK, bool mk) { return mk ? R * (BK + 8) : BK * (R + 8); }

__device__ __forceinline__ void cp16(void *dst, const void *src, bool on) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = on ? 16 : 0;  // 0: the 16 bytes are zero-filled, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <bool T>
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], const bf16 *p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  if constexpr (T)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// One operand tile of R (the output dimension) x BK.  MK: memory rows run
// along the output dimension (row stride ld, k contiguous), kept as
// [R][BK + 8]; otherwise memory rows run along k, kept as [BK][R + 8].
// Everything outside (lim, klim) reads as zero; both are multiples of 8.
template <int R, int BK, bool MK>
__device__ __forceinline__ void load_tile(bf16 *t, const bf16 *__restrict__ g, int ld, int r0, int lim, int k0,
                                          int klim) {
#pragma unroll
  for (int i = 0; i < R * BK / 8 / 128; ++i) {
    const int c = threadIdx.x + i * 128;
    if constexpr (MK) {
      const int r = c / (BK / 8), k = c % (BK / 8) * 8;
      const bool on = r0 + r < lim && k0 + k < klim;
      cp16(t + r * (BK + 8) + k, on ? g + (size_t)(r0 + r) * ld + k0 + k : g, on);
    } else {
      const int k = c / (R / 8), r = c % (R / 8) * 8;
      const bool on = r0 + r < lim && k0 + k < klim;
      cp16(t + k * (R + 8) + r, on ? g + (size_t)(k0 + k) * ld + r0 + r : g, on);
    }
  }
}

// acc = A B over all K for the 32 FM x 64 tile at (m0, n0), one chain of k in
// ascending steps of 16: warp (wm, wn) owns 16 FM x 32 as FM x 4 fragments of
// 16 x 8.  TA: A is stored [K x M]; TB: B is stored [N x K].  ST slices of BK
// in shared memory.
template <int FM, int BK, int ST, bool TA, bool TB>
__device__ __forceinline__ void tile_product(bf16 *sm, float (&acc)[FM][4][4], int M, int N, int m0, int n0, int K,
                                             const bf16 *__restrict__ A, int lda,
                                             const bf16 *__restrict__ B, int ldb) {
  constexpr int BM = 32 * FM, EA = tile_elems(BM, BK, !TA), EB = tile_elems(kBN, BK, TB);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * 16 * FM, wn = (warp & 1) * 32;
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
  const int nk = (K + BK - 1) / BK;
  auto fetch = [&](int it) {
    if (it < nk) {
      bf16 *t = sm + (it % ST) * (EA + EB);
      load_tile<BM, BK, !TA>(t, A, lda, m0, M, it * BK, K);
      load_tile<kBN, BK, TB>(t + EA, B, ldb, n0, N, it * BK, K);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < ST - 1; ++i) fetch(i);
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");
    __syncthreads();  // slice `it` has arrived, and everyone is done with slice it - 1
    fetch(it + ST - 1);
    const bf16 *ta = sm + (it % ST) * (EA + EB), *tb = ta + EA;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      unsigned a[FM][4], b[2][4];
#pragma unroll
      for (int i = 0; i < FM; ++i) {
        // lanes 0-15 address rows 0-15 at k, lanes 16-31 the same rows at k + 8
        if constexpr (!TA)
          ldsm4<false>(a[i], ta + (wm + 16 * i + (lane & 15)) * (BK + 8) + kk + (lane >> 4) * 8);
        else
          ldsm4<true>(a[i], ta + (kk + (lane & 7) + (lane >> 4) * 8) * (BM + 8) + wm + 16 * i + ((lane >> 3) & 1) * 8);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {  // 16 columns: two 8-wide fragments of (k, k + 8)
        if constexpr (!TB)
          ldsm4<true>(b[j], tb + (kk + (lane & 15)) * (kBN + 8) + wn + 16 * j + (lane >> 4) * 8);
        else
          ldsm4<false>(b[j], tb + (wn + 16 * j + (lane & 7) + (lane >> 4) * 8) * (BK + 8) + kk + ((lane >> 3) & 1) * 8);
      }
#pragma unroll
      for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float *c = acc[i][j];
          const unsigned b0 = b[j >> 1][(j & 1) * 2], b1 = b[j >> 1][(j & 1) * 2 + 1];
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
              "{%0,%1,%2,%3};\n"
              : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
              : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b0), "r"(b1));
        }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// The accumulator pairs of this thread: f(row, col, i, j, h) for elements
// (row, col) and (row, col + 1), which are acc[i][j][2 h] and [2 h + 1].
template <int FM, class F>
__device__ __forceinline__ void for_pairs(int m0, int n0, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        f(m0 + (warp >> 1) * 16 * FM + 16 * i + 8 * h + (lane >> 2), n0 + (warp & 1) * 32 + 8 * j + (lane & 3) * 2, i, j, h);
}

// Forward layer, output Z = X W + b.  MODE 0: hidden layer, X' = bf16(silu(Z))
// and Z kept when the backward pass will want it (Zout not null); 1: output
// layer of an evaluation, y on the valid rows and columns; 2: output layer of
// a training step, the errors y - t (Zout) and the gradient of the mean squared
// error 2 (y - t) / (rows n_out) as bf16, both zero on padding columns.
template <int MODE>
__global__ void __launch_bounds__(128) layer_forward(int M, int N, int K, const bf16 *__restrict__ X,
                                                     const bf16 *__restrict__ W, const float *__restrict__ bias,
                                                     float *__restrict__ Zout, bf16 *__restrict__ Xout, int n,
                                                     int n_out, const float *__restrict__ t, float *__restrict__ y) {
  __shared__ __align__(16) bf16 sm[kStages * (tile_elems(kBM, kBK, true) + tile_elems(kBN, kBK, false))];
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  float acc[2][4][4];
  tile_product<2, kBK, kStages, false, false>(sm, acc, M, N, m0, n0, K, X, K, W, N);
  const float scale = MODE == 2 ? 2.0f / ((float)n * (float)n_out) : 0.0f;
  for_pairs<2>(m0, n0, [&](int r, int c, int i, int j, int h) {
    if (r >= M || c >= N) return;
    float z[2] = {acc[i][j][2 * h] + bias[c], acc[i][j][2 * h + 1] + bias[c + 1]};
    if constexpr (MODE == 0) {
      if (Zout) *reinterpret_cast<float2 *>(Zout + (size_t)r * N + c) = make_float2(z[0], z[1]);
      *reinterpret_cast<__nv_bfloat162 *>(Xout + (size_t)r * N + c) =
          __halves2bfloat162(__float2bfloat16(silu(z[0])), __float2bfloat16(silu(z[1])));
    } else if constexpr (MODE == 1) {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (r < n && c + e < n_out) y[(size_t)r * n_out + c + e] = z[e];
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e) z[e] = c + e < n_out ? z[e] - t[(size_t)r * n_out + c + e] : 0.0f;
      *reinterpret_cast<float2 *>(Zout + (size_t)r * N + c) = make_float2(z[0], z[1]);
      *reinterpret_cast<__nv_bfloat162 *>(Xout + (size_t)r * N + c) =
          __halves2bfloat162(__float2bfloat16(scale * z[0]), __float2bfloat16(scale * z[1]));
    }
  });
}

// A row's squared error, as 128 threads sum it: thread c the columns c, c + 128,
// ..., the 32 threads of each of four warps in a tree, the warps in order.
__device__ __forceinline__ float row_error(const float *__restrict__ e, int n_out) {
  const int lane = threadIdx.x & 31;
  float s = 0.0f;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    float sq = 0.0f;
    for (int c = 32 * w + lane; c < n_out; c += 128) sq = fmaf(e[c], e[c], sq);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    s += sq;
  }
  return s;
}

constexpr int kErrRows = 4;  // rows of a block of row errors

// Input gradient of a layer (K inputs, N outputs): dZ W^T (M x K) times
// silu'(Z) of the layer below, as bf16 for the next products and in FP32 in
// Z's place for the bias gradient.  With the last layer, blocks from nb on sum
// the squared errors of kErrRows rows each.
__global__ void __launch_bounds__(128) layer_backward(int M, int N, int K, const bf16 *__restrict__ dZ,
                                                      const bf16 *__restrict__ W, float *__restrict__ Z,
                                                      bf16 *__restrict__ dZin, int nb,
                                                      const float *__restrict__ err, int n_err, int n_out,
                                                      float *__restrict__ row_sq) {
  __shared__ __align__(16) bf16 sm[kStages * (tile_elems(kBM, kBK, true) + tile_elems(kBN, kBK, true))];
  if ((int)blockIdx.x >= nb) {
    for (int i = threadIdx.x >> 5; i < kErrRows; i += 4) {
      const int r = ((int)blockIdx.x - nb) * kErrRows + i;
      if (r >= M) break;
      const float s = row_error(err + (size_t)r * n_err, n_out);
      if ((threadIdx.x & 31) == 0) row_sq[r] = s;
    }
    return;
  }
  float acc[2][4][4];
  const int tk = (K + kBN - 1) / kBN, m0 = (int)blockIdx.x / tk * kBM, n0 = (int)blockIdx.x % tk * kBN;
  tile_product<2, kBK, kStages, false, true>(sm, acc, M, K, m0, n0, N, dZ, N, W, N);
  for_pairs<2>(m0, n0, [&](int r, int c, int i, int j, int h) {
    if (r >= M || c >= K) return;
    float2 *zp = reinterpret_cast<float2 *>(Z + (size_t)r * K + c);
    const float zz[2] = {zp->x, zp->y};
    float g[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float s = 1.0f / (1.0f + expf(-zz[e]));
      g[e] = acc[i][j][2 * h + e] * s * (1.0f + zz[e] * (1.0f - s));
    }
    *zp = make_float2(g[0], g[1]);
    *reinterpret_cast<__nv_bfloat162 *>(dZin + (size_t)r * K + c) =
        __halves2bfloat162(__float2bfloat16(g[0]), __float2bfloat16(g[1]));
  });
}

constexpr int kGradM = 32, kGradK = 64, kGradStages = 3;  // tiles of the weight gradients
constexpr int kColN = 32, kColRows = 64, kColStages = 5;  // of the bias gradients
constexpr size_t kGradBytes = std::max(
    kGradStages * (tile_elems(kGradM, kGradK, false) + tile_elems(kBN, kGradK, false)) * sizeof(bf16),
    kColStages * kColRows * kColN * sizeof(float));

// What the gradients of every layer are summed from.
struct GradArgs {
  int layers, rows;
  int first_w[kMlpMaxLayers + 1], first_b[kMlpMaxLayers + 1];  // first block of each layer
  int K[kMlpMaxLayers], N[kMlpMaxLayers];
  const bf16 *X[kMlpMaxLayers], *dZ[kMlpMaxLayers];
  const float *dZf[kMlpMaxLayers];  // the last: errors, to be scaled
  float *gw[kMlpMaxLayers], *gb[kMlpMaxLayers];
  float scale;
  const float *row_sq;
  float *loss;
};

// Sums of kColN columns over the rows in order: a warp adds, all fetch ahead.
__device__ __forceinline__ void column_sums(float *sm, int rows, int N, int c0, const float *__restrict__ a,
                                            bool scaled, float scale, float *__restrict__ out) {
  const int nt = (rows + kColRows - 1) / kColRows;
  auto fetch = [&](int it) {
    if (it < nt) {
      float *t = sm + (it % kColStages) * kColRows * kColN;
#pragma unroll
      for (int i = 0; i < kColRows * kColN / 4 / 128; ++i) {
        const int q = threadIdx.x + i * 128, r = q / (kColN / 4), c = q % (kColN / 4) * 4;
        const bool on = it * kColRows + r < rows && c0 + c < N;
        cp16(t + r * kColN + c, on ? a + (size_t)(it * kColRows + r) * N + c0 + c : a, on);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kColStages - 1; ++i) fetch(i);
  float s = 0.0f;
  for (int it = 0; it < nt; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kColStages - 2) : "memory");
    __syncthreads();
    fetch(it + kColStages - 1);
    if (threadIdx.x < kColN) {
      const float *t = sm + (it % kColStages) * kColRows * kColN + threadIdx.x;
      float v[kColRows];
#pragma unroll
      for (int u = 0; u < kColRows; ++u) v[u] = t[u * kColN];
#pragma unroll
      for (int u = 0; u < kColRows; ++u) s = __fadd_rn(s, scaled ? __fmul_rn(scale, v[u]) : v[u]);  // (+ 0 past the end)
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (threadIdx.x < kColN && c0 + (int)threadIdx.x < N) out[c0 + threadIdx.x] = s;
}

// All gradients of a training step: weight gradient tiles X^T dZ of every layer
// first (the longest), then columns of the bias gradients, and the last block
// the loss, as 256 threads sum the rows' errors: thread i the rows i, i + 256,
// ..., warps in trees, then in order.
__global__ void __launch_bounds__(128) all_gradients(GradArgs p) {
  __shared__ __align__(16) unsigned char smem[kGradBytes];
  const int b = blockIdx.x, tid = threadIdx.x;
  if (b == p.first_b[p.layers]) {
    float *red = reinterpret_cast<float *>(smem);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float s = 0.0f;
#pragma unroll 4
      for (int r = tid + 128 * h; r < p.rows; r += 256) s += p.row_sq[r];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((tid & 31) == 0) red[4 * h + (tid >> 5)] = s;
    }
    __syncthreads();
    if (tid == 0) {
      float t = 0.0f;
      for (int w = 0; w < 8; ++w) t += red[w];
      *p.loss = t;
    }
    return;
  }
  int l = 0;
  if (b >= p.first_b[0]) {
    while (b >= p.first_b[l + 1]) ++l;
    column_sums(reinterpret_cast<float *>(smem), p.rows, p.N[l], (b - p.first_b[l]) * kColN, p.dZf[l],
                l == p.layers - 1, p.scale, p.gb[l]);
    return;
  }
  while (b >= p.first_w[l + 1]) ++l;
  const int K = p.K[l], N = p.N[l], tn = (N + kBN - 1) / kBN, rest = b - p.first_w[l];
  const int k0 = rest / tn * kGradM, n0 = rest % tn * kBN;
  float acc[1][4][4];
  tile_product<1, kGradK, kGradStages, true, false>(reinterpret_cast<bf16 *>(smem), acc, K, N, k0, n0, p.rows, p.X[l], K,
                                            p.dZ[l], N);
  float *out = p.gw[l];
  for_pairs<1>(k0, n0, [&](int r, int c, int i, int j, int h) {
    if (r < K && c < N)
      *reinterpret_cast<float2 *>(out + (size_t)r * N + c) = make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  });
}

// Adam (Kingma & Ba 2015) on the FP32 master copy; refreshes the BF16 copy
// (the first nw parameters: the weights)
__global__ void adam_step(long n, long nw, float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                          float *__restrict__ v, float lr, float b1, float b2, float eps, float c1,
                          float c2, bf16 *__restrict__ wb) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  if (i < nw) wb[i] = __float2bfloat16(wi);
}

__global__ void to_bf16(long n, const float *__restrict__ a, bf16 *__restrict__ b) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = __float2bfloat16(a[i]);
}

inline int pad16(int x) { return (x + 15) / 16 * 16; }
inline int tiles(int x, int t) { return (x + t - 1) / t; }

inline unsigned blocks(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

Mlp::Mlp(int n_in, int hidden, int layers, int n_out, unsigned long long seed)
    : n_in_(n_in), n_out_(n_out) {
  dims_.push_back(pad16(n_in));
  for (int l = 0; l < layers; ++l) dims_.push_back(pad16(hidden));
  dims_.push_back(pad16(n_out));
  const int L = (int)dims_.size() - 1;
  woff_.assign(L + 1, 0);
  boff_.assign(L + 1, 0);
  for (int l = 0; l < L; ++l) {
    woff_[l + 1] = woff_[l] + (long)dims_[l] * dims_[l + 1];
    boff_[l + 1] = boff_[l] + dims_[l + 1];
  }
  nw_ = woff_[L];
  nb_ = boff_[L];
  // Kaiming-uniform weights on the real fan-in, zero padding rows/columns
  std::mt19937_64 rng(seed);
  std::vector<float> w(nw_, 0.0f), b(nb_, 0.0f);
  for (int l = 0; l < L; ++l) {
    const int fan_in = l == 0 ? n_in : hidden;
    const int kin = l == 0 ? n_in : hidden, kout = l == L - 1 ? n_out : hidden;
    const float bound = std::sqrt(6.0f / (float)fan_in) * (l == L - 1 ? 0.1f : 1.0f);
    std::uniform_real_distribution<float> U(-bound, bound);
    for (int i = 0; i < kin; ++i)
      for (int j = 0; j < kout; ++j) w[woff_[l] + (long)i * dims_[l + 1] + j] = U(rng);
  }
  auto ck = [](cudaError_t e) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("mlp: ") + cudaGetErrorString(e));
  };
  const size_t np = nw_ + nb_;
  ck(cudaMalloc(&master_, np * sizeof(float)));
  ck(cudaMalloc(&grad_, np * sizeof(float)));
  ck(cudaMalloc(&m1_, np * sizeof(float)));
  ck(cudaMalloc(&m2_, np * sizeof(float)));
  ck(cudaMalloc(&wbf_, nw_ * sizeof(bf16)));
  ck(cudaMemset(m1_, 0, np * sizeof(float)));
  ck(cudaMemset(m2_, 0, np * sizeof(float)));
  ck(cudaMemset(grad_, 0, np * sizeof(float)));
  set_params(w.data(), b.data());
}

Mlp::~Mlp() {
  cudaFree(master_);
  cudaFree(grad_);
  cudaFree(m1_);
  cudaFree(m2_);
  cudaFree(wbf_);
  cudaFree(ws_);
}

void Mlp::set_params(const float *w, const float *b) {
  cudaMemcpy(master_, w, nw_ * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemcpy(master_ + nw_, b, nb_ * sizeof(float), cudaMemcpyHostToDevice);
  to_bf16<<<blocks(nw_, 256), 256>>>(nw_, master_, (bf16 *)wbf_);
  cudaDeviceSynchronize();
}

void Mlp::get_params(float *w, float *b) const {
  cudaMemcpy(w, master_, nw_ * sizeof(float), cudaMemcpyDeviceToHost);
  cudaMemcpy(b, master_ + nw_, nb_ * sizeof(float), cudaMemcpyDeviceToHost);
}

void Mlp::get_grads(float *w, float *b) const {
  cudaMemcpy(w, grad_, nw_ * sizeof(float), cudaMemcpyDeviceToHost);
  cudaMemcpy(b, grad_ + nw_, nb_ * sizeof(float), cudaMemcpyDeviceToHost);
}

// Workspace for `rows` rows (a multiple of 16): the bf16 input of every layer
// and a training step's pre-activations, loss gradients of every layer, errors
// and rows' squared errors.  (All of it for an evaluation too: any call of the
// same size then finds its workspace, also one being captured, where nothing
// can be allocated.)
cudaError_t Mlp::carve(int rows, Work &w) {
  const int L = (int)dims_.size() - 1;
  for (int pass = 0; pass < 2; ++pass) {  // sizes, then pointers
    size_t used = 0;
    auto take = [&](size_t bytes) {
      char *q = pass ? (char *)ws_ + used : nullptr;
      used += (bytes + 255) / 256 * 256;
      return q;
    };
    for (int l = 0; l < L; ++l) w.X[l] = (bf16 *)take((size_t)rows * dims_[l] * sizeof(bf16));
    for (int l = 1; l <= L; ++l) w.Z[l] = (float *)take((size_t)rows * dims_[l] * sizeof(float));
    for (int l = 1; l <= L; ++l) w.dZ[l] = (bf16 *)take((size_t)rows * dims_[l] * sizeof(bf16));
    w.row_sq = (float *)take((size_t)rows * sizeof(float));
    if (pass == 0 && used > ws_bytes_) {
      cudaFree(ws_);
      ws_ = nullptr;
      ws_bytes_ = 0;
      const cudaError_t e = cudaMalloc(&ws_, used);
      if (e != cudaSuccess) return e;
      ws_bytes_ = used;
    }
  }
  return cudaSuccess;
}

// The input and the hidden layers (keep: their pre-activations too).
cudaError_t Mlp::hidden_layers(int n, int rows, const float *x, const Work &w, bool keep, cudaStream_t s) {
  // rows beyond n read no input: clear the padded tail of the bf16 input
  if (rows > n) cudaMemsetAsync(w.X[0] + (size_t)n * dims_[0], 0, (size_t)(rows - n) * dims_[0] * sizeof(bf16), s);
  input_to_bf16<<<blocks((long)n * dims_[0], 256), 256, 0, s>>>(n, n_in_, dims_[0], x, w.X[0]);
  for (int l = 0; l + 2 < (int)dims_.size(); ++l) {
    const dim3 grid(tiles(dims_[l + 1], kBN), tiles(rows, kBM));
    layer_forward<0><<<grid, 128, 0, s>>>(rows, dims_[l + 1], dims_[l], w.X[l], (const bf16 *)wbf_ + woff_[l],
                                          master_ + nw_ + boff_[l], keep ? w.Z[l + 1] : nullptr, w.X[l + 1], n, 0,
                                          nullptr, nullptr);
  }
  return cudaGetLastError();
}

cudaError_t Mlp::forward(int n, const float *x, float *y, cudaStream_t s) {
  const int rows = pad16(std::max(n, 1)), L = (int)dims_.size() - 1;
  Work w;
  cudaError_t e = carve(rows, w);
  if (e != cudaSuccess || (e = hidden_layers(n, rows, x, w, false, s)) != cudaSuccess) return e;
  layer_forward<1><<<dim3(tiles(dims_[L], kBN), tiles(rows, kBM)), 128, 0, s>>>(
      rows, dims_[L], dims_[L - 1], w.X[L - 1], (const bf16 *)wbf_ + woff_[L - 1], master_ + nw_ + boff_[L - 1],
      nullptr, nullptr, n, n_out_, nullptr, y);
  return cudaGetLastError();
}

// Forward + backward on one batch (rows a multiple of 16, rows == n): the
// gradient of the mean squared error lands in grad_; returns the loss sum in
// *loss_dev (device float).
cudaError_t Mlp::backward(int n, const float *x, const float *t, float *loss_dev, cudaStream_t s) {
  if (n % 16) return cudaErrorInvalidValue;
  const int L = (int)dims_.size() - 1;
  Work w;
  cudaError_t e = carve(n, w);
  if (e != cudaSuccess || (e = hidden_layers(n, n, x, w, true, s)) != cudaSuccess) return e;
  layer_forward<2><<<dim3(tiles(dims_[L], kBN), tiles(n, kBM)), 128, 0, s>>>(
      n, dims_[L], dims_[L - 1], w.X[L - 1], (const bf16 *)wbf_ + woff_[L - 1], master_ + nw_ + boff_[L - 1], w.Z[L],
      w.dZ[L], n, n_out_, t, nullptr);
  for (int l = L - 1; l > 0; --l) {
    const int nb = tiles(n, kBM) * tiles(dims_[l], kBN);
    layer_backward<<<nb + (l == L - 1 ? tiles(n, kErrRows) : 0), 128, 0, s>>>(
        n, dims_[l + 1], dims_[l], w.dZ[l + 1], (const bf16 *)wbf_ + woff_[l], w.Z[l], w.dZ[l], nb, w.Z[L], dims_[L],
        n_out_, w.row_sq);
  }
  GradArgs p{};
  p.layers = L;
  p.rows = n;
  p.scale = 2.0f / ((float)n * (float)n_out_);
  p.row_sq = w.row_sq;
  p.loss = loss_dev;
  int block = 0;
  for (int l = 0; l < L; ++l) {
    p.K[l] = dims_[l];
    p.N[l] = dims_[l + 1];
    p.X[l] = w.X[l];
    p.dZ[l] = w.dZ[l + 1];
    p.dZf[l] = w.Z[l + 1];
    p.gw[l] = grad_ + woff_[l];
    p.gb[l] = grad_ + nw_ + boff_[l];
    p.first_w[l] = block;
    block += tiles(dims_[l], kGradM) * tiles(dims_[l + 1], kBN);
  }
  p.first_w[L] = block;
  for (int l = 0; l < L; ++l) {
    p.first_b[l] = block;
    block += tiles(dims_[l + 1], kColN);
  }
  p.first_b[L] = block;
  all_gradients<<<block + 1, 128, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t Mlp::adam(float lr, float b1, float b2, float eps, cudaStream_t s) {
  ++step_;
  const float c1 = 1.0f - std::pow(b1, (float)step_), c2 = 1.0f - std::pow(b2, (float)step_);
  adam_step<<<blocks(nw_ + nb_, 256), 256, 0, s>>>(nw_ + nb_, nw_, master_, grad_, m1_, m2_, lr, b1, b2, eps, c1,
                                                   c2, (bf16 *)wbf_);
  return cudaGetLastError();
}

MlpDev Mlp::device_view() const {
  MlpDev d{};
  d.layers = (int)dims_.size() - 1;
  for (int l = 0; l <= d.layers && l <= kMlpMaxLayers; ++l) d.dims[l] = dims_[l];
  for (int l = 0; l < d.layers && l < kMlpMaxLayers; ++l) {
    d.w[l] = (const bf16 *)wbf_ + woff_[l];
    d.b[l] = master_ + nw_ + boff_[l];
  }
  d.n_in = n_in_;
  d.n_out = n_out_;
  return d;
}

}  // namespace zrk

using namespace zrk;

extern "C" {

int zrk_mlp_create(int n_in, int hidden, int layers, int n_out, unsigned long long seed, zrk_mlp_t *out) {
  if (!out) return set_error(ZRK_ERR_INVALID_POINTER, "null output");
  if (n_in < 1 || hidden < 1 || layers < 1 || layers > kMlpMaxLayers - 1 || n_out < 1 || hidden > 1024 ||
      n_in > 1024 || n_out > 1024)
    return set_error(ZRK_ERR_INVALID_ARGUMENT, "mlp sizes out of range");
  try {
    *out = reinterpret_cast<zrk_mlp_t>(new Mlp(n_in, hidden, layers, n_out, seed));
  } catch (const std::exception &e) {
    return set_error(ZRK_ERR_CUDA, e.what());
  }
  return ZRK_OK;
}

int zrk_mlp_free(zrk_mlp_t m) {
  delete reinterpret_cast<Mlp *>(m);
  return ZRK_OK;
}

int zrk_mlp_sizes(zrk_mlp_t m, long *n_weights, long *n_biases) {
  if (!m) return set_error(ZRK_ERR_INVALID_HANDLE, "null mlp");
  Mlp *p = reinterpret_cast<Mlp *>(m);
  if (n_weights) *n_weights = p->n_weights();
  if (n_biases) *n_biases = p->n_biases();
  return ZRK_OK;
}

int zrk_mlp_get_params(zrk_mlp_t m, float *w, float *b) {
  if (!m || !w || !b) return set_error(ZRK_ERR_INVALID_POINTER, "null argument");
  reinterpret_cast<Mlp *>(m)->get_params(w, b);
  return ZRK_OK;
}

int zrk_mlp_set_params(zrk_mlp_t m, const float *w, const float *b) {
  if (!m || !w || !b) return set_error(ZRK_ERR_INVALID_POINTER, "null argument");
  reinterpret_cast<Mlp *>(m)->set_params(w, b);
  return ZRK_OK;
}

int zrk_mlp_get_grads(zrk_mlp_t m, float *w, float *b) {
  if (!m || !w || !b) return set_error(ZRK_ERR_INVALID_POINTER, "null argument");
  cudaDeviceSynchronize();
  reinterpret_cast<Mlp *>(m)->get_grads(w, b);
  return ZRK_OK;
}

int zrk_mlp_forward(zrk_mlp_t m, int n, const float *x, float *y, void *stream) {
  if (!m || !x || !y) return set_error(ZRK_ERR_INVALID_POINTER, "null argument");
  if (n < 0) return set_error(ZRK_ERR_INVALID_ARGUMENT, "n < 0");
  if (n == 0) return ZRK_OK;
  cudaError_t e = reinterpret_cast<Mlp *>(m)->forward(n, x, y, (cudaStream_t)stream);
  return e == cudaSuccess ? ZRK_OK : cuda_error(e, "mlp forward");
}

int zrk_mlp_gradients(zrk_mlp_t m, int n, const float *x, const float *t, float *loss_sum_dev, void *stream) {
  if (!m || !x || !t || !loss_sum_dev) return set_error(ZRK_ERR_INVALID_POINTER, "null argument");
  if (n <= 0 || n % 16) return set_error(ZRK_ERR_INVALID_ARGUMENT, "batch must be a positive multiple of 16");
  cudaError_t e = reinterpret_cast<Mlp *>(m)->backward(n, x, t, loss_sum_dev, (cudaStream_t)stream);
  return e == cudaSuccess ? ZRK_OK : cuda_error(e, "mlp backward");
}

int zrk_mlp_adam(zrk_mlp_t m, float lr, float beta1, float beta2, float eps, void *stream) {
  if (!m) return set_error(ZRK_ERR_INVALID_HANDLE, "null mlp");
  cudaError_t e = reinterpret_cast<Mlp *>(m)->adam(lr, beta1, beta2, eps, (cudaStream_t)stream);
  return e == cudaSuccess ? ZRK_OK : cuda_error(e, "mlp adam");
}

}  // extern "C"
