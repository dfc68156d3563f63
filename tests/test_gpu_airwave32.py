"""The complex64 airwave's line transforms (csrc/k_airlines.cu) against the complex128 oracle
at each length a side can have, more and fewer rows than a CTA takes, and sizes that stay with two-dimensional transforms (two lengths, other lengths, more
rows than the uniform grid). Bound 2e-5 of the largest value, that of every complex64 operator
here; the transforms' own error is about 2^-24 times the 20 roundings of 1024 points."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import oracle_for, probe, product_grid, relerr
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu

# n1fft, n2fft; core nx, ny, nz, nb
CASES = [(256, 256, 29, 12, 4, 2), (1024, 1024, 62, 9, 3, 2), (1024, 1024, 2, 37, 4, 1),
         (64, 64, 2, 2, 3, 1), (64, 256, 29, 12, 4, 2), (256, 1024, 11, 13, 3, 2), (1024, 64, 62, 9, 3, 2),
         (1024, 256, 13, 36, 4, 1), (64, 64, 5, 60, 3, 2), (64, 48, 9, 8, 3, 2), (100, 64, 9, 8, 3, 2)]


@pytest.mark.parametrize("case", CASES, ids=["x".join(map(str, c)) for c in CASES])
def test_airwave_matches_oracle(gpu, tmp_path, case):
    N1, N2, nx, ny, nz, nb = case
    cfg = synthetic.random_small(94, nx=nx, ny=ny, nz=nz, nb=nb, airbc=1, fvm=0, n1fft=N1, n2fft=N2)
    synthetic.write_config(cfg, str(tmp_path))
    p = {k: str(v) for k, v in dict(cfg.params, nb=nb).items()}
    G = product_grid(str(tmp_path), p)
    ctx, O = cs.Ctx(G, 1, 0), oracle_for(G, p)
    O.set_hy_length(False)  # keep Hy and Hz apart where n2 < n3, as the kernel does
    for q, f in enumerate((0.5, 0.75)):
        x, iom = probe(ctx.lE, 5 + q), cs.iom_of(f)
        O.set_iom(iom)
        got, want = ctx.fdfd_apply(iom, x, c64=True), O.fdfd(x)
        assert relerr(got, want) <= 2e-5
        n1, n2 = ctx.n1, ctx.n2  # the rows that the airwave enters, against their own largest
        for o, n in ((0, n1 * (n2 + 1)), (ctx.lEx, (n1 + 1) * n2)):
            assert relerr(got[o:o + n], want[o:o + n]) <= 2e-5
