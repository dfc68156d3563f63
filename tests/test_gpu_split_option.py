"""lusgs_split takes every value, as the switch that it was: 0 the one-pass sweeps, 1 the row
pipeline, any other the default."""
import numpy as np
import pytest

import demo_matrixfree_csem_gb300 as cs
from cases import probe
from demo_matrixfree_csem_gb300 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [-1, 2, 3, 2 ** 31 - 1])
def test_values_other_than_0_and_1_are_the_default(gpu, tmp_path, value):
    ctx = cs.Ctx(synthetic.build_grid(synthetic.random_small(4, 9, 8, 7, airbc=0, nb=2), str(tmp_path)), 0, 0)
    x, iom = probe(ctx.lE, 3), cs.iom_of(0.75)
    want = ctx.lusgs_apply(iom, x, c64=True)
    for v in (0, 1):
        ctx.set_option("lusgs_split", v)
        assert np.abs(ctx.lusgs_apply(iom, x, c64=True) - want).max() <= 1e-6 * np.abs(want).max()
    ctx.set_option("lusgs_split", value)
    assert np.array_equal(ctx.lusgs_apply(iom, x, c64=True), want)
