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
//   * bias, SiLU, its derivative, the loss gradient and the bias-gradient
//     column sums work on the accumulators, so no pass re-reads an output;
//   * the weight gradient, whose output has only 16 tiles, is split over the
//     batch rows into partial sums that one kernel adds in a fixed order, and
//     shares its launch with the input gradient of the same layer.
// 163-256-256-256-161 on a B200: eight training steps at batch 4096, a forward
// pass of 5,001 rows and the copy of the parameters to the host took 15.3 ms
// with a kernel for each elementwise pass, products straight from global
// memory and one block per weight-gradient tile, and take 1.11 ms now.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

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
constexpr int kPadK = kBK + 8, kPadM = kBM + 8;  // padded rows: ldmatrix without bank conflicts
constexpr int kTileElems = kBM * kPadK;          // >= kBK * kPadM
static_assert(kBK * kPadM <= kTileElems && kBM == kBN, "operand tile size");

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

// One operand tile of 64 (the output dimension) x kBK.  MK: memory rows run
// along the output dimension (row stride ld, k contiguous), kept as
// [64][kPadK]; otherwise memory rows run along k, kept as [kBK][kPadM].
// Everything outside (lim, klim) reads as zero; both are multiples of 8.
template <bool MK>
__device__ __forceinline__ void load_tile(bf16 *t, const bf16 *__restrict__ g, int ld, int r0, int lim, int k0,
                                          int klim) {
#pragma unroll
  for (int i = 0; i < kBM * kBK / 8 / 128; ++i) {
    const int c = threadIdx.x + i * 128;
    if constexpr (MK) {
      const int r = c / (kBK / 8), k = c % (kBK / 8) * 8;
      const bool on = r0 + r < lim && k0 + k < klim;
      cp16(t + r * kPadK + k, on ? g + (size_t)(r0 + r) * ld + k0 + k : g, on);
    } else {
      const int k = c / (kBM / 8), r = c % (kBM / 8) * 8;
      const bool on = r0 + r < lim && k0 + k < klim;
      cp16(t + k * kPadM + r, on ? g + (size_t)(k0 + k) * ld + r0 + r : g, on);
    }
  }
}

// acc = A B over k in [k0, k1) for the 64 x 64 tile at (m0, n0): warp (wm, wn)
// owns 32 x 32 as 2 x 4 fragments of 16 x 8.  TA: A is stored [K x M]; TB: B
// is stored [N x K].
template <bool TA, bool TB>
__device__ __forceinline__ void tile_product(bf16 *sm, float (&acc)[2][4][4], int M, int N, int m0, int n0, int k0,
                                             int k1, const bf16 *__restrict__ A, int lda,
                                             const bf16 *__restrict__ B, int ldb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
  const int nk = (k1 - k0 + kBK - 1) / kBK;
  auto fetch = [&](int it) {
    if (it < nk) {
      bf16 *t = sm + (it % kStages) * 2 * kTileElems;
      load_tile<!TA>(t, A, lda, m0, M, k0 + it * kBK, k1);
      load_tile<TB>(t + kTileElems, B, ldb, n0, N, k0 + it * kBK, k1);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) fetch(i);
  for (int it = 0; it < nk; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // slice `it` has arrived, and everyone is done with slice it - 1
    fetch(it + kStages - 1);
    const bf16 *ta = sm + (it % kStages) * 2 * kTileElems, *tb = ta + kTileElems;
#pragma unroll
    for (int kk = 0; kk < kBK; kk += 16) {
      unsigned a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        // lanes 0-15 address rows 0-15 at k, lanes 16-31 the same rows at k + 8
        if constexpr (!TA)
          ldsm4<false>(a[i], ta + (wm + 16 * i + (lane & 15)) * kPadK + kk + (lane >> 4) * 8);
        else
          ldsm4<true>(a[i], ta + (kk + (lane & 7) + (lane >> 4) * 8) * kPadM + wm + 16 * i + ((lane >> 3) & 1) * 8);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {  // 16 columns: two 8-wide fragments of (k, k + 8)
        if constexpr (!TB)
          ldsm4<true>(b[j], tb + (kk + (lane & 15)) * kPadM + wn + 16 * j + (lane >> 4) * 8);
        else
          ldsm4<false>(b[j], tb + (wn + 16 * j + (lane & 7) + (lane >> 4) * 8) * kPadK + kk + ((lane >> 3) & 1) * 8);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
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
  __syncthreads();  // the caller may reuse the operand slices
}

// The accumulator pairs of this thread: f(row, col, i, j, h) for elements
// (row, col) and (row, col + 1), which are acc[i][j][2 h] and [2 h + 1].
template <class F>
__device__ __forceinline__ void for_pairs(int m0, int n0, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        f(m0 + (warp >> 1) * 32 + 16 * i + 8 * h + (lane >> 2), n0 + (warp & 1) * 32 + 8 * j + (lane & 3) * 2, i, j, h);
}

// Column sums of the tile (its rows are the batch rows m0 .. m0 + 63) into
// part[blockrow][N]: over the fragments of a thread, the eight row lanes, the
// two warps of a column half, always in that order.
__device__ __forceinline__ void tile_colsum(float *sm, const float (&v)[2][4][4], int N, int n0, float *part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float s = (v[0][j][e] + v[0][j][e + 2]) + (v[1][j][e] + v[1][j][e + 2]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane < 4) sm[(warp >> 1) * kBN + (warp & 1) * 32 + 8 * j + lane * 2 + e] = s;
    }
  __syncthreads();
  if (threadIdx.x < kBN && n0 + (int)threadIdx.x < N) part[n0 + threadIdx.x] = sm[threadIdx.x] + sm[kBN + threadIdx.x];
}

// Forward layer, output Z = X W + b.  MODE 0: hidden layer, X' = bf16(silu(Z))
// and Z kept when the backward pass will want it (Zout not null); 1: output
// layer of an evaluation, y on the valid rows and columns; 2: output layer of
// a training step, the gradient of the mean squared error 2 (y - t) / (rows
// n_out) as bf16 (zero on padding columns), its column sums (the bias
// gradient of this block of rows) and this tile's squared error.
template <int MODE>
__global__ void __launch_bounds__(128) layer_forward(int M, int N, int K, const bf16 *__restrict__ X,
                                                     const bf16 *__restrict__ W, const float *__restrict__ bias,
                                                     float *__restrict__ Zout, bf16 *__restrict__ Xout, int n,
                                                     int n_out, const float *__restrict__ t, float *__restrict__ y,
                                                     float *__restrict__ db_part, float *__restrict__ loss_part) {
  __shared__ __align__(16) bf16 sm[kStages * 2 * kTileElems];
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  float acc[2][4][4];
  tile_product<false, false>(sm, acc, M, N, m0, n0, 0, K, X, K, W, N);
  float sq = 0.0f;
  const float scale = MODE == 2 ? 2.0f / ((float)n * (float)n_out) : 0.0f;
  for_pairs(m0, n0, [&](int r, int c, int i, int j, int h) {
    float z[2] = {0.0f, 0.0f};
    const bool on = r < M && c < N;
    if (on) {
      z[0] = acc[i][j][2 * h] + bias[c];
      z[1] = acc[i][j][2 * h + 1] + bias[c + 1];
    }
    if constexpr (MODE == 0) {
      if (on) {
        if (Zout) *reinterpret_cast<float2 *>(Zout + (size_t)r * N + c) = make_float2(z[0], z[1]);
        *reinterpret_cast<__nv_bfloat162 *>(Xout + (size_t)r * N + c) =
            __halves2bfloat162(__float2bfloat16(silu(z[0])), __float2bfloat16(silu(z[1])));
      }
    } else if constexpr (MODE == 1) {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (r < n && c + e < n_out) y[(size_t)r * n_out + c + e] = z[e];
    } else {
      float g[2] = {0.0f, 0.0f};
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (on && c + e < n_out) {
          const float d = z[e] - t[(size_t)r * n_out + c + e];
          sq += d * d;
          g[e] = scale * d;
        }
      if (on)
        *reinterpret_cast<__nv_bfloat162 *>(Xout + (size_t)r * N + c) =
            __halves2bfloat162(__float2bfloat16(g[0]), __float2bfloat16(g[1]));
      acc[i][j][2 * h] = g[0];
      acc[i][j][2 * h + 1] = g[1];
    }
  });
  if constexpr (MODE == 2) {
    float *red = reinterpret_cast<float *>(sm);
    tile_colsum(red, acc, N, n0, db_part + (size_t)blockIdx.y * N);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) red[2 * kBN + (threadIdx.x >> 5)] = sq;
    __syncthreads();
    if (threadIdx.x == 0)
      loss_part[blockIdx.y * gridDim.x + blockIdx.x] =
          (red[2 * kBN] + red[2 * kBN + 1]) + (red[2 * kBN + 2] + red[2 * kBN + 3]);
  }
}

// Backward layer l: the first nw blocks form the partial weight gradients
// X^T dZ (K x N) over slices of `chunk` batch rows, the rest the input
// gradient dZ W^T (M x K) times silu'(Z) of the layer below, with its column
// sums.  Both only read dZ, so they run side by side in one launch.
__global__ void __launch_bounds__(128) layer_backward(int M, int N, int K, int nw, int chunk,
                                                      const bf16 *__restrict__ X, const bf16 *__restrict__ dZ,
                                                      float *__restrict__ dW_part, const bf16 *__restrict__ W,
                                                      const float *__restrict__ Zin, bf16 *__restrict__ dZin,
                                                      float *__restrict__ db_part) {
  __shared__ __align__(16) bf16 sm[kStages * 2 * kTileElems];
  float acc[2][4][4];
  if ((int)blockIdx.x < nw) {
    const int tn = (N + kBN - 1) / kBN, tk = (K + kBM - 1) / kBM;
    const int slice = blockIdx.x / (tn * tk), rest = blockIdx.x % (tn * tk);
    const int k0 = rest / tn * kBM, n0 = rest % tn * kBN;
    const int r0 = slice * chunk, r1 = min(M, r0 + chunk);
    tile_product<true, false>(sm, acc, K, N, k0, n0, r0, r1, X, K, dZ, N);
    float *out = dW_part + (size_t)slice * K * N;
    for_pairs(k0, n0, [&](int r, int c, int i, int j, int h) {
      if (r < K && c < N)
        *reinterpret_cast<float2 *>(out + (size_t)r * N + c) = make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
    });
    return;
  }
  const int tk = (K + kBN - 1) / kBN, b = blockIdx.x - nw;
  const int m0 = b / tk * kBM, n0 = b % tk * kBN;
  tile_product<false, true>(sm, acc, M, K, m0, n0, 0, N, dZ, N, W, N);
  for_pairs(m0, n0, [&](int r, int c, int i, int j, int h) {
    float g[2] = {0.0f, 0.0f};
    if (r < M && c < K) {
      const float2 z = *reinterpret_cast<const float2 *>(Zin + (size_t)r * K + c);
      const float zz[2] = {z.x, z.y};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float s = 1.0f / (1.0f + expf(-zz[e]));
        g[e] = acc[i][j][2 * h + e] * s * (1.0f + zz[e] * (1.0f - s));
      }
      *reinterpret_cast<__nv_bfloat162 *>(dZin + (size_t)r * K + c) =
          __halves2bfloat162(__float2bfloat16(g[0]), __float2bfloat16(g[1]));
    }
    acc[i][j][2 * h] = g[0];
    acc[i][j][2 * h + 1] = g[1];
  });
  tile_colsum(reinterpret_cast<float *>(sm), acc, K, n0, db_part + (size_t)(m0 / kBM) * K);
}

// Where the partial sums of every layer's gradient are.
struct GradParts {
  int layers;
  int slices[kMlpMaxLayers];               // partial weight gradients
  long woff[kMlpMaxLayers + 1], boff[kMlpMaxLayers + 1];
  const float *w[kMlpMaxLayers], *b[kMlpMaxLayers];
};

// grad = the partial sums added in slice order (weights; four at a time, the
// layers are multiples of 256 weights) and in block-row order (biases); the
// last block adds the loss of the tiles.
__global__ void __launch_bounds__(256) sum_parts(GradParts p, int blockrows, long nw, long nb, float *__restrict__ grad,
                                                 int ntiles, const float *__restrict__ loss_part,
                                                 float *__restrict__ loss) {
  if (blockIdx.x == gridDim.x - 1) {
    float s = 0.0f;
    for (int i = threadIdx.x; i < ntiles; i += 256) s += loss_part[i];
    __shared__ float red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      float t = 0.0f;
      for (int w = 0; w < 8; ++w) t += red[w];
      *loss = t;
    }
    return;
  }
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (i < nw / 4) {
    int l = 0;
    while (l + 1 < p.layers && 4 * i >= p.woff[l + 1]) ++l;
    const long at = 4 * i - p.woff[l], stride = p.woff[l + 1] - p.woff[l];
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int k = 0; k < p.slices[l]; ++k) {
      const float4 v = *reinterpret_cast<const float4 *>(p.w[l] + k * stride + at);
      s.x += v.x;
      s.y += v.y;
      s.z += v.z;
      s.w += v.w;
    }
    *reinterpret_cast<float4 *>(grad + 4 * i) = s;
  } else if (i - nw / 4 < nb) {
    const long q = i - nw / 4;
    int l = 0;
    while (l + 1 < p.layers && q >= p.boff[l + 1]) ++l;
    const long at = q - p.boff[l], stride = p.boff[l + 1] - p.boff[l];
    float s = 0.0f;
#pragma unroll 8
    for (int k = 0; k < blockrows; ++k) s += p.b[l][k * stride + at];
    grad[nw + q] = s;
  }
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
inline int tiles(int x) { return (x + kBM - 1) / kBM; }

// Slices of the batch rows for a weight gradient of K x N: enough blocks to
// fill the chip (16 output tiles alone would leave 9 of 10 SMs idle), at
// least 64 rows each.
constexpr int kSplitTarget = 148;
inline int split_rows(int rows, int K, int N, int &chunk) {
  const int t = tiles(K) * tiles(N);
  int s = std::min((kSplitTarget + t - 1) / t, std::max(1, rows / 64));
  chunk = (rows + s - 1) / s;
  chunk = (chunk + kBK - 1) / kBK * kBK;
  return (rows + chunk - 1) / chunk;
}
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
// and, for a training step, the pre-activations, the loss gradients of two
// adjacent layers and the partial gradients.
cudaError_t Mlp::carve(int rows, bool train, Work &w) {
  const int L = (int)dims_.size() - 1, br = tiles(rows);
  int maxd = 0;
  for (int d : dims_) maxd = std::max(maxd, d);
  for (int pass = 0; pass < 2; ++pass) {  // sizes, then pointers
    size_t used = 0;
    auto take = [&](size_t bytes) {
      char *q = pass ? (char *)ws_ + used : nullptr;
      used += (bytes + 255) / 256 * 256;
      return q;
    };
    for (int l = 0; l < L; ++l) w.X[l] = (bf16 *)take((size_t)rows * dims_[l] * sizeof(bf16));
    if (train) {
      for (int l = 1; l < L; ++l) w.Z[l] = (float *)take((size_t)rows * dims_[l] * sizeof(float));
      for (auto &d : w.dZ) d = (bf16 *)take((size_t)rows * maxd * sizeof(bf16));
      for (int l = 0; l < L; ++l) {
        w.slices[l] = split_rows(rows, dims_[l], dims_[l + 1], w.chunk[l]);
        w.dW[l] = (float *)take((size_t)w.slices[l] * dims_[l] * dims_[l + 1] * sizeof(float));
        w.db[l] = (float *)take((size_t)br * dims_[l + 1] * sizeof(float));
      }
      w.loss = (float *)take((size_t)br * tiles(dims_[L]) * sizeof(float));
    }
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
    const dim3 grid(tiles(dims_[l + 1]), tiles(rows));
    layer_forward<0><<<grid, 128, 0, s>>>(rows, dims_[l + 1], dims_[l], w.X[l], (const bf16 *)wbf_ + woff_[l],
                                          master_ + nw_ + boff_[l], keep ? w.Z[l + 1] : nullptr, w.X[l + 1], n, 0,
                                          nullptr, nullptr, nullptr, nullptr);
  }
  return cudaGetLastError();
}

cudaError_t Mlp::forward(int n, const float *x, float *y, cudaStream_t s) {
  const int rows = pad16(std::max(n, 1)), L = (int)dims_.size() - 1;
  Work w;
  cudaError_t e = carve(rows, false, w);
  if (e != cudaSuccess || (e = hidden_layers(n, rows, x, w, false, s)) != cudaSuccess) return e;
  layer_forward<1><<<dim3(tiles(dims_[L]), tiles(rows)), 128, 0, s>>>(
      rows, dims_[L], dims_[L - 1], w.X[L - 1], (const bf16 *)wbf_ + woff_[L - 1], master_ + nw_ + boff_[L - 1],
      nullptr, nullptr, n, n_out_, nullptr, y, nullptr, nullptr);
  return cudaGetLastError();
}

// Forward + backward on one batch (rows a multiple of 16, rows == n): the
// gradient of the mean squared error lands in grad_; returns the loss sum in
// *loss_dev (device float).
cudaError_t Mlp::backward(int n, const float *x, const float *t, float *loss_dev, cudaStream_t s) {
  if (n % 16) return cudaErrorInvalidValue;
  const int L = (int)dims_.size() - 1, br = tiles(n);
  Work w;
  cudaError_t e = carve(n, true, w);
  if (e != cudaSuccess || (e = hidden_layers(n, n, x, w, true, s)) != cudaSuccess) return e;
  layer_forward<2><<<dim3(tiles(dims_[L]), br), 128, 0, s>>>(
      n, dims_[L], dims_[L - 1], w.X[L - 1], (const bf16 *)wbf_ + woff_[L - 1], master_ + nw_ + boff_[L - 1],
      nullptr, w.dZ[(L - 1) & 1], n, n_out_, t, nullptr, w.db[L - 1], w.loss);
  GradParts p{};
  p.layers = L;
  p.woff[L] = nw_;
  p.boff[L] = nb_;
  for (int l = L - 1; l >= 0; --l) {
    const int K = dims_[l], N = dims_[l + 1];
    const int nw = w.slices[l] * tiles(K) * tiles(N), na = l > 0 ? br * tiles(K) : 0;
    layer_backward<<<nw + na, 128, 0, s>>>(n, N, K, nw, w.chunk[l], w.X[l], w.dZ[l & 1], w.dW[l],
                                           (const bf16 *)wbf_ + woff_[l], l > 0 ? w.Z[l] : nullptr, w.dZ[(l & 1) ^ 1],
                                           l > 0 ? w.db[l - 1] : nullptr);
    p.slices[l] = w.slices[l];
    p.woff[l] = woff_[l];
    p.boff[l] = boff_[l];
    p.w[l] = w.dW[l];
    p.b[l] = w.db[l];
  }
  sum_parts<<<blocks(nw_ / 4 + nb_, 256) + 1, 256, 0, s>>>(p, br, nw_, nb_, grad_, br * tiles(dims_[L]), w.loss,
                                                           loss_dev);
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
