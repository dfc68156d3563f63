"""complex64 A-phi with its edge sweeps by lines (csrc/k_lusgs6.cu) against the sweeps by diagonals
(<= 1e-6 of the largest value: the same update with sigma grad v in the right-hand side instead of
beside the couplings) and the complex128 oracle (<= 2e-5), on either side of a strip and with few
rows; and not depending on what the output held."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import oracle_for, probe, product_grid, relerr
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("airbc,fvm", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("shape", [(2, 2, 2, 1), (29, 3, 30, 2), (30, 36, 4, 2), (61, 5, 38, 2)], ids=lambda s: "x".join(map(str, s)))
def test_line_edges_match_diagonal_edges_and_oracle(gpu, tmp_path, shape, airbc, fvm):
    nx, ny, nz, nb = shape
    cfg = synthetic.random_small(99, nx=nx, ny=ny, nz=nz, nb=nb, airbc=airbc, fvm=fvm, n1fft=64, n2fft=64)
    synthetic.write_config(cfg, str(tmp_path))
    p = {k: str(v) for k, v in dict(cfg.params, nb=nb).items()}
    G = product_grid(str(tmp_path), p)
    ctx, O = cs.Ctx(G, airbc, fvm), oracle_for(G, p)
    x, iom = probe(ctx.lE, 5), cs.iom_of(0.75)
    O.set_iom(iom)
    got = ctx.aphi_apply(iom, x, c64=True)
    ctx.aphi_apply(iom, np.full_like(x, complex(np.nan, np.inf)), c64=True)
    assert np.array_equal(ctx.aphi_apply(iom, x, c64=True), got)
    ctx.set_option("lusgs_split", 0)
    want = ctx.aphi_apply(iom, x, c64=True)
    assert relerr(got, want) <= 1e-6
    assert relerr(got, O.aphi(x)) <= 2e-5
