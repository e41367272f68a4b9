"""The kernels' interleaved exponentials, logarithms and quotients
(zerork_b200/csrc/kinetics_dev.cuh) and the series of a rate's change with
temperature (kinetics_kernel.cuh) against extended precision.

Bounds: the exponential's polynomial is truncated at 4e-18, its argument
reduction and the last two roundings cost at most one unit in the last place;
a logarithm's three roundings of its leading parts at most two;
a quotient corrected by its residual is within one unit (of the smallest
number, when it underflows), and outside the fast range it is the language's
division, bit for bit.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, have_gpu

pytestmark = pytest.mark.gpu

SRC = r"""
#include "kinetics_dev.cuh"
__global__ void k(int n, const double *a, const double *d, double *e, double *q, double *l) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x[1] = {a[i]}, y[1] = {d[i]};
  double z[1];
  zrk::exps<1>(x, z);
  e[i] = z[0];
  zrk::quotients<1>(x, y, z);
  q[i] = z[0];
  zrk::logs<1>(x, z);
  l[i] = z[0];
}
__global__ void k3(int n, const double *a, const double *d, double *q) {
  const int i = 3 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i + 2 >= n) return;
  const double x[3] = {a[i], a[i + 1], a[i + 2]}, y[3] = {d[i], d[i + 1], d[i + 2]};
  double z[3];
  zrk::quotients<3>(x, y, z);
  for (int j = 0; j < 3; ++j) q[i + j] = z[j];
}
extern "C" int run3(int n, const double *a, const double *d, double *q) {
  k3<<<(n / 3 + 255) / 256, 256>>>(n, a, d, q);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run(int n, const double *a, const double *d, double *e, double *q, double *l) {
  k<<<(n + 255) / 256, 256>>>(n, a, d, e, q, l);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if not have_gpu():
        pytest.skip("no CUDA device")
    import torch
    from zerork_b200 import build
    d = tmp_path_factory.mktemp("exp")
    src, so = str(d / "probe.cu"), str(d / "probe.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc(), "-shared", "-o", so, src] + build._flags(src), check=True)
    lib = C.CDLL(so)

    def run(a, den):
        t = [torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda() for x in (a, den, a, a, a)]
        assert lib.run(len(a), *[C.c_void_p(x.data_ptr()) for x in t]) == 0
        return [x.cpu().numpy() for x in t[2:]]

    def three(a, den):
        t = [torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda() for x in (a, den, a)]
        assert lib.run3(len(a), *[C.c_void_p(x.data_ptr()) for x in t]) == 0
        return t[2].cpu().numpy()

    run.three = three
    return run


def _ulps(x, exact):
    return float(np.max(np.abs(x.astype(np.longdouble) - exact) / np.spacing(np.abs(exact).astype(np.float64))))


@pytest.mark.parametrize("lo,hi", [(-1e-6, 1e-6), (-1.0, 1.0), (-50.0, 50.0), (-700.0, 709.0)])
def test_exp(probe, lo, hi):
    x = np.random.default_rng(1).uniform(lo, hi, 200001)
    e, _, _ = probe(x, np.ones_like(x))
    assert _ulps(e, np.exp(x.astype(np.longdouble))) <= 1.0


def test_exp_ends(probe):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 709.78, 709.79, 1e300, -1e300, -745.0, -746.0, -720.0, 750.0])
    e, _, _ = probe(x, np.ones_like(x))
    with np.errstate(over="ignore", under="ignore"):
        r = np.exp(x)
    assert np.array_equal(np.isnan(e), np.isnan(r)) and np.array_equal(np.isinf(e), np.isinf(r))
    ok = np.isfinite(r)
    assert np.all(np.abs(e[ok] - r[ok]) <= np.maximum(np.spacing(r[ok]), 5e-324))


def test_logs(probe):
    r = np.random.default_rng(3)
    x = np.concatenate([2.0 ** r.uniform(-1020, 1020, 100001), r.uniform(0.4, 2.5, 100001), 1.0 + r.uniform(-1e-6, 1e-6, 9999)])
    _, _, l = probe(x, np.ones_like(x))
    assert _ulps(l, np.log(x.astype(np.longdouble))) <= 2.0
    x = np.array([1.0, 0.0, -1.0, np.inf, np.nan, 5e-324, 1e-310])
    _, _, l = probe(x, np.ones_like(x))
    with np.errstate(all="ignore"):
        assert np.allclose(l, np.log(x), rtol=4e-16, atol=0.0, equal_nan=True)


@pytest.mark.parametrize("span", [10, 499, 720, 1020])
def test_quotients(probe, span):
    r = np.random.default_rng(2)
    a = r.choice([-1.0, 1.0], 200001) * 2.0 ** r.uniform(-span, span, 200001)
    d = r.choice([-1.0, 1.0], 200001) * 2.0 ** r.uniform(-span, span, 200001)
    exact = a.astype(np.longdouble) / d.astype(np.longdouble)
    with np.errstate(all="ignore"):
        ref = a / d
    over = np.isinf(ref)
    for q in (probe(a, d)[1], probe.three(a, d)):
        assert np.array_equal(q[over], ref[over])
        assert np.all(np.abs(q - exact)[~over] <= np.maximum(np.spacing(np.abs(ref[~over])), 5e-324))


def test_quotient_ends(probe):
    ends = np.array([0.0, -0.0, 1.0, 5e-324, 1e-310, 1e-250, 1e250, 1.7e308, np.inf, -np.inf, np.nan])
    a, d = (x.ravel() for x in np.meshgrid(ends, ends))
    _, q, _ = probe(a, d)
    with np.errstate(all="ignore"):
        assert np.array_equal(q, a / d, equal_nan=True)
    # one argument out of range sends all of a group the language's way
    mixed = np.repeat(np.array([[3.0, 7.0, 1.0]]), len(a), axis=0), np.repeat(np.array([[7.0, 3.0, 1.0]]), len(a), axis=0)
    for j in range(3):
        x, y = mixed[0].copy(), mixed[1].copy()
        x[:, j], y[:, j] = a, d
        with np.errstate(all="ignore"):
            assert np.allclose(probe.three(x.ravel(), y.ravel()), (x / y).ravel(), rtol=2.3e-16, atol=0.0, equal_nan=True)


CHANGE = r"""
#include "kinetics_kernel.cuh"
__global__ void k(int n, const double *x, const double *w, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  zrk::RxnRec R = {};
  R.n = 1.0;  // the exponent is dlogT
  R.rev = -1;
  R.nr = 1;
  const double c[1] = {1.0}, dl[1] = {x[i]}, di[1] = {0.0};
  double rop[1] = {w[i]};  // the limited constant over a limit of 1
  out[i] = zrk::rop_change<1, 1>(R, 0, c, c, rop, dl, di, w[i] > 0.0 ? 1.0 : 0.0) ? rop[0] : -1.0;
}
extern "C" int run(int n, const double *x, const double *w, double *out) {
  k<<<(n + 255) / 256, 256>>>(n, x, w, out);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.parametrize("w", [1e-9, 0.1, 0.5, 0.9, 0.999])
def test_rate_change(tmp_path, w):
    """e (1 - w) / (1 + w e) w, e = expm1(x), over all |x| that the series take
    (below 1e-4; beyond, the rate is left alone).  Truncation 1e-16 and six
    roundings."""
    if not have_gpu():
        pytest.skip("no CUDA device")
    import torch
    from zerork_b200 import build
    src, so = str(tmp_path / "change.cu"), str(tmp_path / "change.so")
    with open(src, "w") as f:
        f.write(CHANGE)
    subprocess.run([build.nvcc(), "-shared", "-o", so, src] + build._flags(src), check=True)
    x = np.concatenate([np.linspace(-0.999e-4, 0.999e-4, 2000), 10.0 ** np.linspace(-12, -4.01, 500), [1.001e-4, -2e-4]])
    t = [torch.from_numpy(a).cuda() for a in (x, np.full_like(x, w), np.zeros_like(x))]
    assert C.CDLL(so).run(len(x), *[C.c_void_p(a.data_ptr()) for a in t]) == 0
    got = t[2].cpu().numpy()
    assert np.all(got[-2:] == -1.0)
    X, W = x[:-2].astype(np.longdouble), np.longdouble(w)
    e = np.expm1(X)
    exact = e * (1 - W) / (1 + W * e) * W
    assert np.max(np.abs(got[:-2] / exact - 1)) <= 1e-16 + 6 * 2.0 ** -53
