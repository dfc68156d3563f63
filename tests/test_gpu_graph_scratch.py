"""Captured iterations of the batched solver while the sweeps' scratch moves. With the air above the
model, LU-SGS sweeps more planes than A-phi and needs the larger scratch: here 56 row steps a line
against 48 (csrc/k_sweep_common.cuh line_steps), so A-phi first and LU-SGS then moves it. The
iterations captured before must not be replayed on the old address: the same bits as without
graphs."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import product_grid
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algopt", [1, 2])
def test_preconditioners_in_turn_on_one_context(gpu, tmp_path, algopt):
    cfg = synthetic.random_small(57, nx=20, ny=18, nz=40, nb=5, airbc=1, n1fft=64, n2fft=64)
    synthetic.write_config(cfg, str(tmp_path))
    G = product_grid(str(tmp_path), {k: str(v) for k, v in dict(cfg.params, nb=5).items()})
    freqs = np.array([0.5, 0.5, 1.0], np.float32)
    srcs = np.repeat(cfg.acq.src[:1, :3], 3, axis=0)
    srcs[1, 0] += 37.0

    def runs(graphs):
        ctx = cs.Ctx(G, 1, 0)
        ctx.set_option("graphs", graphs)
        # 12 iterations, or 3 cycles of 4: launched, captured, replayed
        return [cs.solve_batch(ctx, freqs, srcs, rec=cfg.acq.rec, precision=32, algopt=algopt, preco=p, niter=12, tol=1e-30,
                               inner_tol=1e-20, max_outer=1, check_every=4, nrestart=4) for p in (3, 1, 3, 1)]

    for got, want in zip(runs(1), runs(0)):
        assert np.array_equal(got["iters"], want["iters"]) and got["iters"].min() >= 4
        assert np.all(np.isfinite(want["dcal"])) and np.array_equal(got["dcal"], want["dcal"])
