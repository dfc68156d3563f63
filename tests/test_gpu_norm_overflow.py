"""<a, a> in complex128 where its sum leaves the finite numbers: what the general product gives (a
copy as the second vector), which is 0 for the imaginary part while no product of a value's two
parts overflows, and NaN from there on. Lengths of one launch and of two, the value in a thread's
first round and in a later one."""
import numpy as np
import pytest

from test_gpu_dots import _dot

pytestmark = pytest.mark.gpu

VALUES = [1e160 + 1j, 1 - 1e160j, 1e154 + 1e154j, 1e200 + 1e200j, complex(np.inf, 0), complex(np.inf, 2), complex(0, -np.inf),
          complex(np.nan, 1), complex(1, np.nan), complex(np.inf, np.nan), 1e300 + 0j]


@pytest.mark.parametrize("n", [1, 700, 2049, 16384, 40000])
def test_norms_that_overflow(gpu, n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    for at in {0, n // 2, n - 1}:
        a = torch.randn((len(VALUES), n), dtype=torch.complex128, device="cuda", generator=gen)
        a[:, at] = torch.tensor(VALUES, dtype=torch.complex128, device="cuda")
        a[0, (at + 5) % n] = 1e160 + 1j  # one more, in another thread
        norm, general = _dot(64, a, a), _dot(64, a, a.clone())
        assert np.array_equal(norm.view(np.float64), general.view(np.float64), equal_nan=True), (at, norm, general)
        assert norm[0].imag == 0 and np.isinf(norm[0].real)
