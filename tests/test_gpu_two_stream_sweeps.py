"""The complex64 schedules that are not the default, selected by lusgs_split, which
test_gpu_grouped_sweeps, test_gpu_tiled_sweeps and test_gpu_parity leave as it is where they set
their own options: lusgs_split 1 (k_lusgs5.cu), where grids too large for the line sweeps go and the
autotuner may, on two streams or one, with capped grids, and 0 (k_lusgs2.cu) with several lines a
CTA. The bounds are those tests' own."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import probe, relerr
from demo_matrixfree_csem_gb300 import api
from test_gpu_grouped_sweeps import FREQS, SHAPES, _lusgs_batch, _setup

pytestmark = pytest.mark.gpu

IDS = [f"{s[1]}x{s[2]}x{s[3]}_air{s[5]}_fvm{s[6]}" for s in SHAPES]


def _launches(f):
    n = api.lib().csem_launch_count()
    return f(), api.lib().csem_launch_count() - n


@pytest.mark.parametrize("shape", SHAPES[:3], ids=IDS[:3])
def test_two_streams_give_the_bits_of_one(gpu, tmp_path, shape):
    cfg, G, ctx, O = _setup(tmp_path, *shape)
    freqs = FREQS + [0.5, 1.0]  # 9 systems: halves of 4 and 5
    X = np.stack([probe(ctx.lE, shape[0] + 30 + q) for q in range(len(freqs))])
    ctx.set_option("lusgs_split", 1)
    ctx.set_option("lusgs_overlap", 0)
    one, n1 = _launches(lambda: _lusgs_batch(ctx, freqs, X))
    ctx.set_option("lusgs_overlap", 1)
    for cap in (4, 1, 0):
        ctx.set_option("lusgs_cap", cap)
        two, n2 = _launches(lambda: _lusgs_batch(ctx, freqs, X))
        assert np.array_equal(one, two), cap
        assert n2 == n1 + 12  # six passes and six pipelines of the second half
    O.set_freq(freqs[3])
    assert relerr(two[3], O.lusgs(X[3])) <= 2e-5


def test_two_streams_in_the_mixed_solve(gpu, tmp_path):
    cfg, G, ctx, O = _setup(tmp_path, *SHAPES[1])
    freqs = np.array([0.5, 0.75, 1.0, 0.5, 0.75, 1.0, 0.5, 0.75, 1.0, 0.5], np.float32)
    src = np.repeat(cfg.acq.src[:1, :3], len(freqs), axis=0)
    src[:, 0] += np.arange(len(freqs), dtype=np.float32) * 29.0
    ctx.set_option("lusgs_split", 1)
    out = {}
    for ov in (0, 1):
        ctx.set_option("lusgs_overlap", ov)
        out[ov] = cs.solve_batch(ctx, freqs, src, rec=cfg.acq.rec, precision=32, preco=1, niter=1000, tol=1e-8)
        assert out[ov]["status"] == ["converged"] * len(freqs), (ov, out[ov]["status"])
    assert np.array_equal(out[0]["dcal"], out[1]["dcal"])
    assert np.array_equal(out[0]["iters"], out[1]["iters"])


@pytest.mark.parametrize("shape", SHAPES + [(61, 12, 290, 9, 4, 0, 0)], ids=IDS + ["12x290x9"])
def test_widths_and_lines_of_the_row_pipelines(gpu, tmp_path, shape):
    cfg, G, ctx, O = _setup(tmp_path, *shape)
    O.set_freq(0.75)
    iom = cs.iom_of(0.75)
    x = probe(ctx.lE, shape[0] + 1)
    mo = O.lusgs(x)
    for split in (0, 1):
        ctx.set_option("lusgs_split", split)
        for vw in (0, 1, 2, 4):
            ctx.set_option("lusgs_vw", vw)
            ctx.set_option("lusgs_lines", 1)
            ref = ctx.lusgs_apply(iom, x, c64=True)
            assert relerr(ref, mo) <= 2e-5, (split, vw)
            for lines in (2, 3, 7) if split == 0 else ():
                ctx.set_option("lusgs_lines", lines)
                got = ctx.lusgs_apply(iom, x, c64=True)
                assert relerr(got, ref) <= 1e-6, (vw, lines, relerr(got, ref))
