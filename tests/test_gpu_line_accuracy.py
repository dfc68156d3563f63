"""Error of the complex64 line sweeps (csrc/k_lusgs6.cu) against complex128, relative, in the
two-norm, beside that of the sweeps that they take the place of, on layered earths without water of
200 x 150 x 100 and 50 x 150 x 100 m cells, where a rounding of the reciprocal spacings, the same
all along a line, shows.

A-phi: the sweeps by diagonals divide, at 2 roundings a quotient; the lines multiply by reciprocals
that are good to the last place, and add one rounding (B) and one product. Both errors are sums of
as many independent roundings of a value, most of them the node sweeps', which are the same code: no
more than 1.25 times. LU-SGS: the row pipeline multiplies by a reciprocal of three roundings, four
with iwmu, and a diagonal of two, all of them the same along a line, the lines by one of half: no
more than it."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [11, 12])
@pytest.mark.parametrize("fvm", [0, 1])
@pytest.mark.parametrize("n,h,nb", [((55, 9, 33), (200.0, 150.0, 100.0), 5), ((7, 39, 23), (50.0, 150.0, 100.0), 4)])
def test_error_of_the_lines(gpu, n, h, nb, fvm, seed):
    rng = np.random.default_rng(seed)
    x = [((np.arange(m + 1) - (m / 2 if a < 2 else 0)) * d).astype(np.float32) for a, (m, d) in enumerate(zip(n, h))]
    rho = np.exp(rng.uniform(0, np.log(5.0), n[2])).astype(np.float32)[:, None, None] * np.ones((1, n[1], n[0]), np.float32)
    ctx = cs.Ctx(cs.Grid.from_arrays(*x, rho, rho, 1.5 * rho).extend(nb, 4e3), 0, fvm)
    v = (rng.standard_normal(ctx.lE) + 1j * rng.standard_normal(ctx.lE)).astype(np.complex64)

    def error(apply, split):
        ctx.set_option("lusgs_split", split)
        errors = []
        for f in (0.25, 1.0):
            want = apply(cs.iom_of(f), v)
            errors.append(np.linalg.norm(apply(cs.iom_of(f), v, c64=True) - want) / np.linalg.norm(want))
        return np.linalg.norm(errors)

    assert error(ctx.aphi_apply, 2) <= 1.25 * error(ctx.aphi_apply, 0)
    assert error(ctx.lusgs_apply, 2) <= error(ctx.lusgs_apply, 1)
