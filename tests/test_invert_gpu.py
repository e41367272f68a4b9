"""The dense integrator's blocked inversion and its product
(zerork_b200/csrc/integrator_dense.cuh) on matrices of every panel remainder,
register-chunk count and CTA size, with the matrix and the pivot order in shared
memory or in global memory (the group path above its limit), against numpy.

Bound: x = (I - cJ)^-1 b from an explicit inverse is within
n eps cond(W^-1 P W) of the solution in the weighted norm; the matrices here
are badly row-scaled (12 decades) before the weights undo it.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import have_gpu

pytestmark = pytest.mark.gpu

SRC = r"""
#include "integrator_dense.cuh"
namespace zrk {
template <class LT>
__global__ void __launch_bounds__(512, 1) probe(DevMech m, int n, int lda, double c, const double *J,
                                                const double *scale, const double *b, double *x, int *bad) {
  extern __shared__ double sm[];
  Smem s;
  double *p = sm;
  s.red = p; p += 128;
  s.rows = p; p += kPanelMax * n;
  s.bs = p; p += n;
  s.wlu = p; p += n;
  s.scale = p; p += n;
  s.perm = (int *)p; p += (n + 1) / 2 + 1;
  s.A = p;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s.scale[i] = scale[i];
  __syncthreads();
  const int r = invert_any<LT, true>((n + 31) / 32, m, s, J, c, n, lda);
  if (threadIdx.x == 0) *bad = r;
  if (!r) apply_inverse<LT>(s, n, lda, b, x);
}
// Matrix and pivot order in global memory; the product by a thread a row.
__global__ void __launch_bounds__(512, 1) probe_global(DevMech m, int n, int lda, double c, const double *J,
                                                       const double *scale, const double *b, double *x, int *bad,
                                                       double *A, int *perm) {
  extern __shared__ double sm[];
  Smem s;
  double *p = sm;
  s.red = p; p += 128;
  s.rows = p; p += panel_width(true, (n + 31) / 32) * n;
  s.bs = p; p += n;
  s.wlu = p; p += n;
  s.scale = p; p += n;
  s.perm = perm;
  s.A = A;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s.scale[i] = scale[i];
  __syncthreads();
  const int r = invert_any<double, false>((n + 31) / 32, m, s, J, c, n, lda);
  if (threadIdx.x == 0) *bad = r;
  if (r) return;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s.bs[pivot_col(s.perm, i)] = b[i] / s.wlu[i];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double a = 0.0;
    for (int j = 0; j < n; ++j) a += A[(size_t)i * lda + j] * s.bs[j];
    const int k = pivot_col(s.perm, i);
    x[k] = a * s.wlu[k];
  }
}
}  // namespace zrk
extern "C" int run_global(int threads, int n, const int *nz_rc, double c, const double *J, const double *scale,
                          const double *b, double *x, int *bad, double *A, int *perm) {
  using namespace zrk;
  DevMech m{};
  m.nnz = n * n;
  m.nz_rc = nz_rc;
  const int smem = (128 + (panel_width(true, (n + 31) / 32) + 3) * n) * 8;
  probe_global<<<1, threads, smem>>>(m, n, n | 1, c, J, scale, b, x, bad, A, perm);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run(int fp32, int threads, int n, const int *nz_rc, double c, const double *J, const double *scale,
                   const double *b, double *x, int *bad) {
  using namespace zrk;
  DevMech m{};
  m.nnz = n * n;
  m.nz_rc = nz_rc;
  const int lda = n | 1;
  const int smem = (128 + (kPanelMax + 3) * n + (n + 1) / 2 + 1) * 8 + n * lda * (fp32 ? 4 : 8);
  const void *k = fp32 ? (const void *)probe<float> : (const void *)probe<double>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 1;
  if (fp32) probe<float><<<1, threads, smem>>>(m, n, lda, c, J, scale, b, x, bad);
  else probe<double><<<1, threads, smem>>>(m, n, lda, c, J, scale, b, x, bad);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if not have_gpu():
        pytest.skip("no CUDA device")
    import torch
    from zerork_b200 import build
    d = tmp_path_factory.mktemp("inv")
    src, so = str(d / "probe.cu"), str(d / "probe.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc(), "-shared", "-o", so, src] + build._flags(src), check=True)
    lib = C.CDLL(so)
    lib.run.argtypes = [C.c_int] * 3 + [C.c_void_p, C.c_double] + [C.c_void_p] * 5
    lib.run_global.argtypes = [C.c_int] * 2 + [C.c_void_p, C.c_double] + [C.c_void_p] * 7

    def run(J, c, scale, b, fp32, threads):
        n = len(b)
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
               ((i | j << 16).astype(np.int32).ravel(), J.ravel(), scale, b, np.zeros(n), np.ones(1, np.int32))]
        p = [C.c_void_p(a.data_ptr()) for a in dev]
        assert lib.run(int(fp32), threads, n, p[0], c, *p[1:]) == 0
        return dev[4].cpu().numpy(), int(dev[5].item())

    def run_global(J, c, scale, b, threads):
        n = len(b)
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
               ((i | j << 16).astype(np.int32).ravel(), J.ravel(), scale, b, np.zeros(n), np.ones(1, np.int32),
                np.zeros(n * (n | 1)), np.zeros(n + 1, np.int32))]
        p = [C.c_void_p(a.data_ptr()) for a in dev]
        assert lib.run_global(threads, n, p[0], c, *p[1:]) == 0
        return dev[4].cpu().numpy(), int(dev[5].item())

    run.in_global = run_global
    return run


@pytest.mark.parametrize("threads", [32, 96, 128, 256, 512])
@pytest.mark.parametrize("fp32,sizes", [(False, (1, 2, 8, 9, 11, 32, 33, 80, 97, 128, 129, 150, 161)),
                                        (True, (7, 16, 65, 127, 160, 161, 193, 220)),
                                        ("global", (3, 97, 161, 192, 193, 197, 224, 225, 256))])
def test_inverse(probe, fp32, sizes, threads):
    in_global, fp32 = fp32 == "global", fp32 is True
    eps = 2.0 ** (-24 if fp32 else -53)
    for n in sizes:
        r = np.random.default_rng(n)
        scale = 10.0 ** r.uniform(-12, 0, n)
        c, M = 1e-3, r.standard_normal((n, n))  # W^-1 P W = 0.1 I + M: pivoting is needed
        Pw = 0.1 * np.eye(n) + M
        J = (np.eye(n) - scale[:, None] * Pw / scale[None, :]) / c
        b = scale * r.standard_normal(n)
        x, bad = probe.in_global(J, c, scale, b, threads) if in_global else probe(J, c, scale, b, fp32, threads)
        assert bad == 0
        ref = np.linalg.solve(Pw, b / scale)
        # I - cJ is formed from J: its rounding enters times the condition
        err = np.linalg.norm(x / scale - ref) / np.linalg.norm(ref)
        assert err <= 8 * n * eps * np.linalg.cond(Pw), (n, err)


def test_singular(probe):
    for n, threads in ((9, 32), (40, 128), (161, 512)):
        r = np.random.default_rng(3)
        Pw = r.standard_normal((n, n))
        Pw[:, n // 2] = 0.0
        for bad_value in (0.0, np.nan, np.inf):
            Q = Pw.copy()
            Q[0, 0] = Q[0, 0] if bad_value == 0.0 else bad_value
            J = np.eye(n) - Q
            if bad_value == 0.0:  # exact zero column after I - J
                J[:, n // 2] = np.eye(n)[:, n // 2]
            assert probe(J, 1.0, np.ones(n), np.ones(n), False, threads)[1] != 0
