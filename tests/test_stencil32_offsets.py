"""The complex64 stencil's byte offsets (csrc/offsets32.h, csrc/k_fdfd32.cu): 32 bits while they
reach every point of a component, 64 beyond.

CPU: every grid that the rule gives 32 bits has its corners at the offsets that 64 bits give, and
the smallest grids that it gives 64 bits to have a point which 32 bits miss.
GPU: A x on a grid whose components hold more than 4 GiB, where the planes near the bottom, past
4 GiB and near the top are, bit for bit, those of grids of a few planes cut out of it."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "demo_matrixfree_csem_gb300", "csrc")

PROGRAM = r"""
#include "offsets32.h"
#include <cstdint>
#include <cstdio>
using namespace csem;
template <class Off> static Off last(int c, int n1, int n2, int n3) {
  const int w = c == 0 ? n1 : n1 + 1, h = c == 1 ? n2 : n2 + 1, d = c == 2 ? n3 : n3 + 1;
  return point_offset<Off>(w - 1, h - 1, d - 1, w, 8 * (Off)w * h);
}
int main() {
  long wrong = 0, narrow = 0, wide = 0;
  const int side[] = {2, 31, 100, 511, 645, 811, 812, 1023, 4095, 20000};
  for (int n1 : side)
    for (int n2 : side) {
      // planes on either side of the largest that 32 bits reach
      const long edge = (long)(536870912.0 / ((n1 + 1.0) * (n2 + 1.0)));
      for (long n3 = edge > 3 ? edge - 3 : 1; n3 <= edge + 3; n3++) {
        bool same = true;
        for (int c = 0; c < 3; c++)
          same = same && (uint64_t)last<uint32_t>(c, n1, n2, (int)n3) == last<uint64_t>(c, n1, n2, (int)n3);
        wrong += same != offsets32_reach(n1, n2, (int)n3);
        (same ? narrow : wide)++;
      }
    }
  printf("%ld %ld %ld\n", wrong, narrow, wide);
}
"""


def test_offsets_where_32_bits_reach(tmp_path):
    src, exe = tmp_path / "off.cpp", tmp_path / "off"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    wrong, narrow, wide = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert wrong == 0 and narrow > 100 and wide > 100


def _grid(d1, d2, d3, sigma):
    """A padded grid of these spacings; sigma, the same array for all three directions."""
    import demo_matrixfree_csem_gb300 as cs
    from demo_matrixfree_csem_gb300 import api
    g = cs.Grid()
    g.keep = [sigma]

    def hold(a):
        g.keep.append(np.ascontiguousarray(a, np.float64))
        return api._p(g.keep[-1])

    for a, d in enumerate((d1, d2, d3), 1):
        n, x = len(d) - 1, np.concatenate([[0.0], np.cumsum(d[:-1])])
        setattr(g.g, f"n{a}", n)
        setattr(g.g, "n" + "xyz"[a - 1], n)
        for nm, v in ((f"x{a}", x), (f"x{a}s", x + 0.5 * d), (f"d{a}", d), (f"d{a}s", 1.01 * d)):
            setattr(g.g, nm, hold(v))
    for nm in ("sigma11", "sigma22", "sigma33"):
        setattr(g.g, nm, api._p(sigma))
    return g


@pytest.mark.gpu
def test_components_of_more_than_4_gib(gpu):
    import ctypes as C

    import torch

    import demo_matrixfree_csem_gb300 as cs
    from demo_matrixfree_csem_gb300 import api
    if torch.cuda.mem_get_info()[0] < 100e9 or os.sysconf("SC_AVPHYS_PAGES") * os.sysconf("SC_PAGE_SIZE") < 60e9:
        pytest.skip("needs 100 GB of device and 60 GB of host memory")
    n1, n2, n3 = 1024, 1023, 530  # Ex: 557 M points, 4.5 GB
    rng = np.random.default_rng(8)
    d1, d2, d3 = (rng.uniform(50.0, 150.0, n + 1) for n in (n1, n2, n3))
    plane = (n1 + 1) * (n2 + 1)  # a plane's conductivities: the same array for all of them
    sigma = np.full(plane * (n3 + 1), 0.25)
    iom = np.array([0.0, cs.iom_of(0.75).imag])

    def apply(ctx, x):
        y = torch.full_like(x, float("nan"))
        torch.cuda.synchronize()
        rc = api.lib().csem_fdfd_apply_dev(ctx.h, 32, 1, api._p(iom), C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), None)
        assert rc == 0, api.lib().csem_last_error().decode()
        torch.cuda.synchronize()
        return y

    def parts(v, n):
        a, b = n1 * (n2 + 1) * (n + 1), (n1 + 1) * n2 * (n + 1)
        return v[:a].view(n + 1, -1), v[a:a + b].view(n + 1, -1), v[a + b:].view(n, -1)

    big = cs.Ctx(_grid(d1, d2, d3, sigma), 0, 0)
    x = torch.randn(big.lE, dtype=torch.complex64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    y = parts(apply(big, x), n3)
    planes = 6
    wrap = 2 ** 29 // (n1 * (n2 + 1))
    for k in (0, wrap - planes // 2, n3 - planes):  # cut out planes k .. k + 6
        cut = cs.Ctx(_grid(d1, d2, d3[k:k + planes + 1], sigma), 0, 0)
        xc = torch.cat([v[k:k + planes + (c < 2)].reshape(-1) for c, v in enumerate(parts(x, n3))])
        want = parts(apply(cut, xc), planes)
        for c in range(3):  # (the planes that a cut makes Ex's and Ey's boundaries are not the grid's)
            lo, hi = (int(k > 0), planes + int(k + planes == n3)) if c < 2 else (0, planes)
            assert torch.equal(y[c][k + lo:k + hi], want[c][lo:hi]), (k, c)
