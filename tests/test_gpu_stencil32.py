"""The complex64 stencil (csrc/k_fdfd32.cu) against the complex128 oracle where it can go
wrong: columns on either side of a tile of 30 and of two, rows on either side of a tile's
height, fewer rows than one, planes on either side of a chunk; with and without air and FVM.
Bound 2e-5 relative (max norm), the bound of every complex64 operator here: a point sums some
ten products rounded to 2^-24, of which the largest can cancel to a twentieth."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import oracle_for, probe, product_grid, relerr
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu

# padded cells n1, n2, nK = core + 2 nb; n1 + 1 columns and n2 + 1 rows of nodes
SHAPES = [(2, 2, 2, 1), (24, 3, 5, 2), (25, 4, 30, 2), (26, 11, 8, 2), (55, 12, 3, 2), (56, 27, 62, 2)]


@pytest.mark.parametrize("airbc,fvm", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_stencil_matches_oracle(gpu, tmp_path, shape, airbc, fvm):
    nx, ny, nz, nb = shape
    cfg = synthetic.random_small(93, nx=nx, ny=ny, nz=nz, nb=nb, airbc=airbc, fvm=fvm, n1fft=64, n2fft=64)
    synthetic.write_config(cfg, str(tmp_path))
    p = {k: str(v) for k, v in dict(cfg.params, nb=nb).items()}
    G = product_grid(str(tmp_path), p)
    ctx, O = cs.Ctx(G, airbc, fvm), oracle_for(G, p)
    O.set_hy_length(False)  # keep Hy and Hz apart where n2 < n3, as the kernel does
    x, iom = probe(ctx.lE, 5), cs.iom_of(0.75)
    O.set_iom(iom)
    want = O.fdfd(x)
    for by in (4, 8, 16):
        ctx.set_option("stencil_by", by)
        assert relerr(ctx.fdfd_apply(iom, x, c64=True), want) <= 2e-5
