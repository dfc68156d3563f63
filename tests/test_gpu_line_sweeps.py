"""complex64 LU-SGS as a pass and a chain with a warp per line (csrc/k_lusgs6.cu, the default
schedule) against the one-pass pipelined sweeps (<= 1e-6, the bound of the other schedules:
the same update up to multiply-add contraction) and the complex128 oracle (<= 2e-5), where it
can go wrong: columns on either side of a strip of 32 and of two, rows on either side of the
shortest strip (40), fewer lines than Ex's CTA takes, rows in the air and below; and batches
whose frequencies' groups hold one system, 16 and 17."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import oracle_for, probe, product_grid, relerr
from demo_matrixfree_csem_gb300 import api, synthetic
from test_gpu_grouped_sweeps import _lusgs_batch

pytestmark = pytest.mark.gpu

# padded cells n1, n2, nK = core + 2 nb; n - 1 columns / rows are swept
SHAPES = [(2, 2, 2, 1), (29, 3, 30, 2), (30, 36, 4, 2), (28, 29, 37, 2), (61, 5, 38, 2), (62, 9, 33, 2), (3, 62, 39, 3)]


def _setup(d, seed, shape, airbc, fvm):
    nx, ny, nz, nb = shape
    cfg = synthetic.random_small(seed, nx=nx, ny=ny, nz=nz, nb=nb, airbc=airbc, fvm=fvm, n1fft=64, n2fft=64)
    synthetic.write_config(cfg, str(d))
    p = {k: str(v) for k, v in dict(cfg.params, nb=nb).items()}
    G = product_grid(str(d), p)
    return cs.Ctx(G, airbc, fvm), oracle_for(G, p)


@pytest.mark.parametrize("airbc,fvm", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_line_sweeps_match_one_pass_sweeps_and_oracle(gpu, tmp_path, shape, airbc, fvm):
    ctx, O = _setup(tmp_path, 91, shape, airbc, fvm)
    freqs = [0.75, 0.5, 0.75]
    X = np.stack([probe(ctx.lE, 5 + q) for q in range(3)])
    got = _lusgs_batch(ctx, freqs, X)
    ctx.set_option("lusgs_split", 0)
    want = _lusgs_batch(ctx, freqs, X)
    for q, f in enumerate(freqs):
        O.set_freq(f)
        assert relerr(got[q], want[q]) <= 1e-6
        assert relerr(got[q], O.lusgs(X[q])) <= 2e-5


@pytest.mark.parametrize("counts", [(1, 16, 2), (17, 1, 1)])
def test_groups_of_any_size_give_each_system_its_own_bits(gpu, tmp_path, counts):
    """A system's result does not depend on the batch it is in: w is the same whether one
    system of the group forms it or another."""
    ctx, _ = _setup(tmp_path, 92, (30, 9, 11, 2), 1, 0)
    freqs = [f for f, n in zip((0.5, 1.0, 0.25), counts) for _ in range(n)]
    freqs = freqs[::2] + freqs[1::2]  # the systems of a frequency apart
    X = np.stack([probe(ctx.lE, 40 + q) for q in range(len(freqs))])
    got = _lusgs_batch(ctx, freqs, X)
    for q, f in enumerate(freqs):
        assert np.array_equal(got[q], _lusgs_batch(ctx, [f], X[q:q + 1])[0])


@pytest.mark.parametrize("shape", [(29, 3, 30, 2), (3, 30, 29, 2)], ids=["29x3x30x2", "3x30x29x2"])
def test_large_batches_give_each_system_its_own_bits(gpu, tmp_path, shape):
    """33 systems: more lines than 7 on each of 152 SMs (chunks of 4 rows), and more of Ex's CTAs
    than SMs (8 lines to a CTA); a system alone takes the other shapes."""
    ctx, _ = _setup(tmp_path, 95, shape, 1, 0)
    freqs = [(0.5, 1.0, 0.25)[q % 3] for q in range(33)]
    X = np.stack([probe(ctx.lE, 60 + q) for q in range(len(freqs))])
    got = _lusgs_batch(ctx, freqs, X)
    for q in (0, 1, 16, 31, 32):
        assert np.array_equal(got[q], _lusgs_batch(ctx, freqs[q:q + 1], X[q:q + 1])[0])


@pytest.mark.parametrize("airbc,fvm", [(0, 0), (1, 1)])
@pytest.mark.parametrize("shape", SHAPES[:4], ids=["x".join(map(str, s)) for s in SHAPES[:4]])
def test_output_of_any_content_is_overwritten(gpu, tmp_path, shape, airbc, fvm):
    """Only the boundary edges of y are cleared beforehand: the rest must not be read."""
    import ctypes as C

    import torch
    ctx, _ = _setup(tmp_path, 96, shape, airbc, fvm)
    x = torch.from_numpy(np.stack([probe(ctx.lE, 7 + q) for q in range(3)]).astype(np.complex64)).cuda()
    z = cs.iom_of(0.75)
    iom = np.array([z.real, z.imag] * 3)
    out = []
    for fill in (0.0, float("nan")):
        y = torch.full_like(x, complex(fill, fill))
        torch.cuda.synchronize()
        assert api.lib().csem_lusgs_apply_dev(ctx.h, 32, 3, iom.ctypes.data_as(C.POINTER(C.c_double)),
                                                 C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), None) == 0
        torch.cuda.synchronize()
        out.append(y.cpu().numpy())
    assert np.isfinite(out[1]).all() and np.array_equal(out[0], out[1])


# rows that are no multiple of 8, march positions in one strip and in several
@pytest.mark.parametrize("shape", [(40, 37, 45, 2), (61, 5, 38, 2), (5, 62, 41, 2), (30, 29, 66, 2)], ids=lambda s: "x".join(map(str, s)))
def test_result_does_not_depend_on_what_the_scratch_holds(gpu, tmp_path, shape):
    """The stream's entries past the last row and position are never written, so they hold another
    component's or another call's values; none may reach a result."""
    freqs = [0.75, 0.5]
    ctx, _ = _setup(tmp_path, 97, shape, 1, 0)
    X = np.stack([probe(ctx.lE, 9 + q) for q in range(2)])
    want = _lusgs_batch(ctx, freqs, X)
    _lusgs_batch(ctx, freqs, np.full_like(X, complex(np.nan, np.inf)))
    assert np.isfinite(want).all() and np.array_equal(_lusgs_batch(ctx, freqs, X), want)
