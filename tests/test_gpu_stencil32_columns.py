"""The complex64 stencil's tiles (csrc/k_fdfd32.cu): 30 columns, and columns 0 and n1 with the first
and the last of them. n1 on either side of one tile and of two, against the complex128 operator, at
the bound of test_gpu_stencil32; every entry is written, and the time of a grid that fills its tiles
is no longer than that of the next larger grid, which takes a tile more."""
import ctypes as C

import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import probe, relerr
from demo_matrixfree_csem_gb300 import api, synthetic

pytestmark = pytest.mark.gpu


def _ctx(tmp_path, n1, n2, n3, airbc, fvm):
    cfg = synthetic.random_small(95, nx=n1 - 2, ny=n2 - 2, nz=n3 - 2, nb=1, airbc=airbc, fvm=fvm, n1fft=64, n2fft=64)
    return cs.Ctx(synthetic.build_grid(cfg, str(tmp_path)), airbc, fvm)


@pytest.mark.parametrize("airbc,fvm", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("n1", [3, 29, 30, 31, 32, 59, 60, 61, 62, 63])
def test_columns_of_one_and_two_tiles(gpu, tmp_path, n1, airbc, fvm):
    import torch
    ctx = _ctx(tmp_path, n1, 11, 9, airbc, fvm)
    assert ctx.n1 == n1
    x, iom = probe(ctx.lE, 5), cs.iom_of(0.75)
    want = ctx.fdfd_apply(iom, x)
    xd = torch.from_numpy(x.astype(np.complex64)).cuda()
    yd = torch.full_like(xd, complex(np.nan, np.nan))
    torch.cuda.synchronize()
    i2 = np.array([iom.real, iom.imag])
    rc = api.lib().csem_fdfd_apply_dev(ctx.h, 32, 1, api._p(i2), C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    got = yd.cpu().numpy().astype(np.complex128)
    assert np.all(np.isfinite(got)) and relerr(got, want) <= 2e-5
    assert np.all(got[want == 0] == 0)  # the boundaries


def test_a_grid_that_fills_its_tiles(gpu, tmp_path):
    import torch
    us = {}
    for n1 in (30, 31, 32):
        ctx = _ctx(tmp_path, n1, 140, 120, 0, 0)
        x = torch.randn(24, ctx.lE, dtype=torch.complex64, device="cuda")
        y = torch.empty_like(x)
        iom = np.zeros(48)
        iom[1::2] = cs.iom_of(0.75).imag
        st = torch.cuda.ExternalStream(ctx.stream)
        torch.cuda.synchronize()
        times = []
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(st)
            for _ in range(4):
                rc = api.lib().csem_fdfd_apply_dev(ctx.h, 32, 24, api._p(iom), C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), None)
                assert rc == 0
            e[1].record(st)
            e[1].synchronize()
            times.append(e[0].elapsed_time(e[1]))
        us[n1] = min(times)
    assert us[30] <= 0.85 * us[32] and us[31] <= 0.85 * us[32], us  # one tile and two
