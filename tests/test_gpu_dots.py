"""Dot products of every length range (csrc/k_blas.cu: one cluster of up to 8 blocks to a vector
in one launch, or two launches) and <a, a> in complex128, which sums the real part alone: against
exact sums, and against the general product bit for bit. Bounds: a sum of n products in pairs
(complex64) or in FP64 by blocks of at most n / 256 terms, 2^-52 n / 256 + 2^-50 of the sum of
absolute products is far below 1e-13 here."""
import numpy as np
import pytest

from demo_matrixfree_csem_gb300 import api

pytestmark = pytest.mark.gpu


def _dot(prec, a, b):
    import ctypes as C

    import torch
    out = torch.zeros(a.shape[0], dtype=torch.complex128, device="cuda")
    rc = api.lib().csem_cdot_dev(prec, C.c_long(a.shape[1]), a.shape[0], C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()),
                                 C.cast(out.data_ptr(), C.POINTER(C.c_double)), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return out.cpu().numpy()


# around a block's 2048 elements, and around 8 blocks
@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 14336, 16383, 16384, 16385, 40000])
@pytest.mark.parametrize("prec", [32, 64])
def test_dots_of_every_length(gpu, prec, n):
    import torch
    dt = torch.complex64 if prec == 32 else torch.complex128
    gen = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randn((3, n), dtype=dt, device="cuda", generator=gen) for _ in range(2))
    x, y = a.cpu().numpy().astype(np.clongdouble), b.cpu().numpy().astype(np.clongdouble)
    got = _dot(prec, a, b)
    assert np.all(np.abs(got - (x * y.conj()).sum(1)) <= 1e-13 * np.abs(x * y).sum(1))
    norm, again = _dot(prec, a, a), _dot(prec, a, a.clone())  # <a, a> knows its argument, a copy does not
    assert np.array_equal(norm.view(np.float64), again.view(np.float64))
