"""Options set between two batched solves on one context, whose iterations are captured: the second
solve runs what a new context with the option runs, bit for bit, and not what the first captured."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import product_grid
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algopt", [1, 2])
@pytest.mark.parametrize("preco,option,values", [(1, "lusgs_split", (2, 1, 0, 2)), (3, "lusgs_split", (2, 1, 2)),
                                                 (3, "aphi_fix", (0, 1, 0)), (1, "lusgs_pipelined", (1, 0))])
def test_options_between_solves(gpu, tmp_path, algopt, preco, option, values):
    cfg = synthetic.random_small(58, nx=22, ny=18, nz=16, nb=4, airbc=0)
    synthetic.write_config(cfg, str(tmp_path))
    G = product_grid(str(tmp_path), {k: str(v) for k, v in dict(cfg.params, nb=4).items()})
    freqs = np.array([0.5, 0.5, 1.0], np.float32)
    srcs = np.repeat(cfg.acq.src[:1, :3], 3, axis=0)
    srcs[1, 0] += 37.0

    def run(ctx, value):
        ctx.set_option(option, value)
        r = cs.solve_batch(ctx, freqs, srcs, rec=cfg.acq.rec, precision=32, algopt=algopt, preco=preco, niter=12, tol=1e-30,
                           inner_tol=1e-20, max_outer=1, check_every=4, nrestart=4)
        assert np.all(np.isfinite(r["dcal"]))
        return r["dcal"]

    one, new = cs.Ctx(G, 0, 0), {}
    for v in values:
        if v not in new:
            ctx = cs.Ctx(G, 0, 0)
            ctx.set_option("graphs", 0)
            new[v] = run(ctx, v)
        assert np.array_equal(run(one, v), new[v]), v
    assert not np.array_equal(new[values[0]], new[values[1]])  # the option is one that shows
