"""Preconditioners with the device nearly full. The complex64 line sweeps' scratch (csrc/k_lusgs6.cu)
is larger than what LU-SGS's split sweeps take, A-phi's sweeps by diagonals take none, nor do those
of complex128, whose pipelines (csrc/k_lusgs64.cu) have a table: where it does not fit, those run,
and give what they give when they are asked for."""
import ctypes as C

import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from demo_matrixfree_csem_gb300 import api, synthetic

pytestmark = pytest.mark.gpu

NSYS = 128
# entries a slot, 16 bytes each: 84 lines of 3 strips of 88 rows of 32; a component's points; A-phi's
# node vectors, which come first, and half the lines'; half the table's
LINES, POINTS, NODES, TABLE = 84 * 3 * 88 * 32, 84 * 85 * 85, 85 ** 3, 3 * 85 * 85


@pytest.mark.parametrize("name,prec,option,value,leave", [
    ("lusgs", 32, "lusgs_split", 1, (LINES + POINTS) // 2), ("aphi", 32, "lusgs_split", 0, NODES + LINES // 2),
    ("lusgs", 64, "lusgs_pipelined", 0, TABLE // 2), ("aphi", 64, "lusgs_pipelined", 0, 2 * NODES + TABLE // 2)])
def test_scratch_that_does_not_fit(gpu, tmp_path, name, prec, option, value, leave):
    import torch
    G = synthetic.build_grid(synthetic.random_small(5, 64, 64, 64, airbc=0, nb=10), str(tmp_path))
    ctx = cs.Ctx(G, 0, 0)
    assert (ctx.n1, ctx.n2, ctx.n3) == (84, 84, 84)
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(NSYS, ctx.lE, dtype=torch.complex64 if prec == 32 else torch.complex128, device="cuda", generator=gen)
    iom = np.zeros(2 * NSYS)
    iom[1::2] = [cs.iom_of(f).imag for f in (0.5, 1.0)] * (NSYS // 2)

    y = torch.empty_like(x)

    def apply(c):
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        rc = getattr(api.lib(), f"csem_{name}_apply_dev")(c.h, prec, NSYS, iom.ctypes.data_as(C.POINTER(C.c_double)),
                                                         C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), None)
        assert rc == 0, api.lib().csem_last_error().decode()
        torch.cuda.synchronize()
        return y

    ctx.set_option(option, value)
    want = apply(ctx).clone()
    del ctx
    assert torch.equal(apply(cs.Ctx(G, 0, 0)), want) == (prec == 64)  # (complex128: the same bits either way)
    ctx = cs.Ctx(G, 0, 0)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - 16 * NSYS * leave, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            assert torch.equal(apply(ctx), want)
    finally:
        del hold, ctx
        torch.cuda.empty_cache()
