"""The complex128 sweeps with two threads a row (csrc/k_lusgs64.cu) and their integer reciprocal.

CPU: xd_den and xd_div2 (csrc/exact_div.h) equal the / operator bit for bit.
GPU: LU-SGS and A-phi equal the one-launch-per-diagonal kernels bit for bit with rows on either
side of what one kernel takes (128, 256), and of a warp."""
import os
import subprocess

import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from demo_matrixfree_csem_gb300 import synthetic

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "demo_matrixfree_csem_gb300", "csrc")

PROGRAM = r"""
#include "exact_div.h"
#include <cstdio>
#include <random>
using namespace csem;
int main() {
  std::mt19937_64 g(11);
  long wrong = 0, missed = 0;
  auto num = [&]() {
    uint64_t m = g() & 0xfffffffffffffull;
    switch (g() % 8) {
      case 0: m &= ~((1ull << (g() % 53)) - 1); break;
      case 1: m |= (1ull << (g() % 53)) - 1; break;
      case 2: m = g() % 16; break;
      case 3: m = 0xfffffffffffffull - g() % 16; break;
    }
    return xd_double((g() & (1ull << 63)) | m | ((640 + g() % 767) << 52));
  };
  for (long i = 0; i < 8000000; i++) {
    const double a = num(), d = num();
    uint32_t bad = 0;
    const XdDen n = xd_den(d, bad);
    const double q = xd_div2(a, d, n.R, bad);
    missed += bad;
    wrong += !bad && xd_bits(q) != xd_bits(a / d);
  }
  printf("%ld %ld\n", wrong, missed);
  return 0;
}
"""


def test_reciprocals_give_the_division_operators_quotients(tmp_path):
    src, exe = tmp_path / "den.cpp", tmp_path / "den"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)])
    assert subprocess.check_output([str(exe)]).split() == [b"0", b"0"]


# padded planes nz + 4: nz + 3 rows of Ex and Ey
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 30, 29), (3, 4, 125), (4, 3, 126), (2, 3, 253), (3, 2, 254)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("airbc,fvm", [(0, 0), (0, 1), (1, 0)])
def test_paired_rows_equal_diagonal_sweeps(gpu, tmp_path, shape, airbc, fvm):
    cfg = synthetic.random_small(8, *shape, airbc=airbc, fvm=fvm, nb=2)
    G = synthetic.build_grid(cfg, str(tmp_path))
    ctx = cs.Ctx(G, airbc, fvm)
    rng = np.random.default_rng(3)
    x = rng.standard_normal(ctx.lE) + 1j * rng.standard_normal(ctx.lE)
    wild = x * 10.0 ** rng.uniform(-320, 150, ctx.lE)  # subnormal and beyond exact_div.h's range
    with np.errstate(all="ignore"):
        for iom in (cs.iom_of(0.75), complex(1e-7, 5e-6)):
            for v in (x, wild):
                for apply in (ctx.lusgs_apply, ctx.aphi_apply):
                    ctx.set_option("lusgs_pipelined", 0)
                    want = apply(iom, v)
                    ctx.set_option("lusgs_pipelined", 1)
                    got = apply(iom, v)
                    assert np.array_equal(got.view(np.float64), want.view(np.float64), equal_nan=True)
