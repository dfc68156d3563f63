"""The complex128 kernels' quotients by integer arithmetic (csrc/exact_div.h).

CPU: xd_div and xd_div2 equal the / operator bit for bit over significands of every shape
(random, short, all ones, near a rounding boundary) and the whole exponent range they
accept; outside it they say so.
GPU: the sweeps that use them equal the one-launch-per-diagonal kernels, which divide with
the / operator, bit for bit, also where operands leave that range (subnormal, huge and
infinite values) or iom has a real part and the kernels fall back."""
import os
import subprocess

import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from demo_matrixfree_csem_gb300 import synthetic

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "demo_matrixfree_csem_gb300", "csrc")

PROGRAM = r"""
#include "exact_div.h"
#include <cmath>
#include <cstdio>
#include <random>
using namespace csem;
int main() {
  std::mt19937_64 g(7);
  long wrong = 0, missed = 0, ok = 0;
  auto num = [&](int spread) {
    uint64_t m = g() & 0xfffffffffffffull;
    switch (g() % 8) {
      case 0: m &= ~((1ull << (g() % 52)) - 1); break;
      case 1: m |= (1ull << (g() % 52)) - 1; break;
      case 2: m = g() % 16; break;
      case 3: m = 0xfffffffffffffull - g() % 16; break;
    }
    return xd_double(m | ((uint64_t)(1023 + (int)(g() % (2 * spread)) - spread) << 52));
  };
  for (long i = 0; i < 8000000; i++) {
    const double d = num(380);
    double a = num(380);
    if (i % 3 == 0) {  // a / d next to the midpoint of two doubles
      const double q = xd_double((g() & 0xfffffffffffffull) | (1023ull << 52));
      a = (double)((long double)q * d + (long double)d * 0x1p-53L);
    }
    if (i % 2) a = -a;
    if (i % 1000 == 0) a = i % 2000 ? 0.0 : -0.0;
    uint32_t bad = 0;
    double r = xd_div(a, d, xd_recip(d), bad);
    const bool in = a == 0 || xd_in_range((uint32_t)(xd_bits(a) >> 32));
    if ((bad == 0) != in) missed++;
    if (!bad && xd_bits(r) != xd_bits(a / d)) wrong++;
    const double dd = g() % 2 ? d : -d;
    const uint64_t R = (xd_bits(d) << 12) == 0 ? ~0ull : ((xd_bits(1.0 / d) & 0xfffffffffffffull) | (1ull << 52)) << 11;
    bad = 0;
    r = xd_div2(a, dd, R, bad);
    if ((bad == 0) != in) missed++;
    if (!bad && r != a / dd) wrong++;
    ok += !bad;
  }
  const double out[] = {1e-310, 1e-200, 1e200, INFINITY, NAN};
  for (double a : out) {
    uint32_t bad = 0;
    xd_div(a, 3.0, xd_recip(3.0), bad);
    missed += bad == 0;
  }
  for (double d : out) missed += xd_recip(d) != 0;
  printf("%ld %ld %ld\n", wrong, missed, ok);
  return 0;
}
"""


def test_quotients_equal_the_division_operator(tmp_path):
    src, exe = tmp_path / "xd.cpp", tmp_path / "xd"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    wrong, missed, ok = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert wrong == 0 and missed == 0 and ok > 7000000


# rows on either side of a warp, of several warps, of the named barriers' 256; 2 rows
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 3, 2), (9, 31, 30), (35, 33, 32), (7, 6, 262)])
@pytest.mark.parametrize("airbc,fvm", [(0, 0), (0, 1), (1, 0)])
def test_pipelined_sweeps_equal_diagonal_sweeps(gpu, tmp_path, shape, airbc, fvm):
    cfg = synthetic.random_small(5, *shape, airbc=airbc, fvm=fvm, nb=2)
    G = synthetic.build_grid(cfg, str(tmp_path))
    ctx = cs.Ctx(G, airbc, fvm)
    rng = np.random.default_rng(3)
    x = rng.standard_normal(ctx.lE) + 1j * rng.standard_normal(ctx.lE)
    sparse = np.where(rng.random(ctx.lE) < 0.9, 0, x)       # zeros, as around a source
    wild = x * 10.0 ** rng.uniform(-320, 150, ctx.lE)       # subnormal and beyond the range
    inf = x.copy()
    inf[ctx.lE // 2] = np.inf
    with np.errstate(all="ignore"):
        for iom in (cs.iom_of(0.75), complex(1e-7, 5e-6)):
            for v in (x, sparse, wild, inf):
                for apply in (ctx.lusgs_apply, ctx.aphi_apply):
                    ctx.set_option("lusgs_pipelined", 0)
                    want = apply(iom, v)
                    ctx.set_option("lusgs_pipelined", 1)
                    got = apply(iom, v)
                    assert np.array_equal(got.view(np.float64), want.view(np.float64), equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("airbc,fvm", [(0, 0), (0, 1)])
def test_operator_equals_oracle(gpu, tmp_path, airbc, fvm):
    """Columns on either side of a 31-wide tile, planes on either side of a chunk."""
    from cases import oracle_for
    cfg = synthetic.random_small(6, 29, 14, 40, airbc=airbc, fvm=fvm, nb=2)
    G = synthetic.build_grid(cfg, str(tmp_path))
    ctx = cs.Ctx(G, airbc, fvm)
    O = oracle_for(G, cfg.params)
    O.set_hy_length(False)  # n2 < n3: keep Hy and Hz apart, as the kernel does
    rng = np.random.default_rng(4)
    x = rng.standard_normal(ctx.lE) + 1j * rng.standard_normal(ctx.lE)
    for v in (x, np.where(rng.random(ctx.lE) < 0.9, 0, x), x * 10.0 ** rng.uniform(-320, 150, ctx.lE)):
        for iom in (cs.iom_of(0.75), complex(1e-7, 5e-6)):
            O.set_iom(iom)
            assert np.array_equal(ctx.fdfd_apply(iom, v), O.fdfd(v))
