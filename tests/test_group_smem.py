"""Shared memory of the plain FP64 group path (zerork_b200/csrc/
integrator_group.h), on the host: what it holds, and where its limits lie."""
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include "integrator_group.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **v) {
  size_t a[6];
  for (int i = 0; i < 6; ++i) a[i] = strtoul(v[i + 1], nullptr, 10);
  const zrk::GroupSmem g = zrk::group_smem(a[0], a[1], a[2], a[3], a[4], a[5]);
  printf("%zu %zu %zu %d %d", g.matrix_at, g.eval, g.fac, g.chunks, g.fac_smem);
}
"""
LIMIT = 227 * 1024 // 8


@pytest.fixture(scope="module")
def smem(tmp_path_factory):
    d = tmp_path_factory.mktemp("smem")
    src, exe = str(d / "g.cu"), str(d / "g")
    with open(src, "w") as f:
        f.write(SRC)
    from zerork_b200 import build
    subprocess.run([build.nvcc(), "-std=c++17", "-I" + build.CSRC, "-I" + ROOT + "/include", "-o", exe, src], check=True)

    def run(nsp, nstep):
        n = nsp + 1
        width = 8 if n <= 128 else 6 if n <= 192 else 4
        args = nsp, nstep, 4 * nsp + 2, width * n, n * (n | 1), LIMIT
        r = subprocess.run([exe] + [str(a) for a in args], check=True, capture_output=True, text=True)
        at, ev, fac, chunks, fs = (int(x) for x in r.stdout.split())
        ws = 128 + 3 * nsp + nstep
        # the pivot rows end before the matrix, the evaluation's parts inside its size
        assert at >= 128 + args[3] and at >= ws and ev >= ws + (args[2] if chunks else 0)
        assert fac >= (at + args[4] if fs else ev) and (not fs or fac <= LIMIT)
        return ev, bool(chunks), bool(fs)

    return run


def test_factorization_stays_in_shared_memory(smem):
    """160 species: with up to 2,527 steps the matrix fits beside the rates
    workspace (128 + 480 + 2527 + 161 x 161 doubles), partial sums or not."""
    assert smem(160, 2527)[2] and not smem(160, 2528)[2]
    assert smem(160, 1886) == (128 + 480 + 1886 + 642, True, True)
    assert smem(10, 27)[2] and smem(1, 2)[2]


def test_what_fits_without_partial_sums_runs(smem):
    """255 species: partial sums up to 27,141 steps, and up to 28,163 steps the
    evaluation fits without them."""
    ev, chunks, _ = smem(255, 27141)
    assert chunks and ev == LIMIT
    ev, chunks, _ = smem(255, 28163)
    assert not chunks and ev == LIMIT
    assert smem(255, 28164)[0] > LIMIT
