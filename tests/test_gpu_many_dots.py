"""Dot products of many short vectors (csrc/k_blas.cu short_dots): one launch up to the number of
vectors from which two are faster, and the same bits on either side."""
import numpy as np
import pytest

from demo_matrixfree_csem_gb300 import api
from test_gpu_dots import _dot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,same,most", [(32, 1000, 0, 128), (64, 1000, 0, 128), (64, 5000, 0, 128), (32, 9000, 0, 76),
                                              (64, 14000, 0, 32), (64, 16384, 0, 14), (64, 16384, 1, 48), (32, 16384, 0, 48)])
def test_vectors_of_one_launch_and_of_two(gpu, prec, n, same, most):
    import torch
    dt = torch.complex64 if prec == 32 else torch.complex128
    gen = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn((300, n), dtype=dt, device="cuda", generator=gen)
    b = a if same else torch.randn((300, n), dtype=dt, device="cuda", generator=gen)
    got = {}
    for m, launches in ((most, 1), (most + 1, 2), (300, 2)):
        before = api.lib().csem_launch_count()
        got[m] = _dot(prec, a[:m], a[:m] if same else b[:m])
        assert api.lib().csem_launch_count() - before == launches, m
    for m in got:
        assert np.array_equal(got[m].view(np.float64), got[300][:m].view(np.float64))
