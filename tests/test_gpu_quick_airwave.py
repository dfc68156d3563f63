"""The complex128 airwave's line transforms (csrc/k_airlines.cu), which the batched solver's outer
residuals take: one outer step's residual with them against the one with the reference's operations
(option quick_residual 0), at every length of a side. The two round differently, by some 2^-53 times
the sum of a row's absolute terms, which is below 1e4 |b| here, and the residual is above 0.01 |b|:
bound 1e-9."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import product_grid
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(64, 5, 4, 6, 2), (256, 29, 12, 6, 2), (1024, 13, 36, 5, 3)], ids=lambda c: "x".join(map(str, c)))
def test_quick_residual_equals_the_exact_one(gpu, tmp_path, case):
    N, nx, ny, nz, nb = case
    cfg = synthetic.random_small(98, nx=nx, ny=ny, nz=nz, nb=nb, airbc=1, n1fft=N, n2fft=N, freqs=(0.5, 1.0))
    synthetic.write_config(cfg, str(tmp_path))
    G = product_grid(str(tmp_path), {k: str(v) for k, v in cfg.params.items()})
    rel = []
    for quick in (0, 1):
        ctx = cs.Ctx(G, 1, 0)
        ctx.set_option("quick_residual", quick)
        r = cs.solve_batch(ctx, [0.5, 0.5, 1.0], np.tile(cfg.acq.src[0], (3, 1)), rec=cfg.acq.rec, precision=32, niter=2,
                           inner_tol=1e-2, max_outer=1)
        rel.append(r["relres"])
    assert np.all(rel[0] > 1e-2) and np.all(np.abs(rel[1] - rel[0]) <= 1e-9 * rel[0])
