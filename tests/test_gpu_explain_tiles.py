"""GkmExplain lookups (gkm_explain_table) at the edges of a block's positions (128 - l
+ 1 of a row) against the sums over each window's neighbours: rows of 117 .. 119 and
235 .. 238 positions, one and no window, padding past a row, l = 6, 8, 11, weighted and
not, all modes.  Both add the same terms; the table's went through transforms of 4^l
values, whose rounding is a few units of 1e-16 per pass of the largest entry: 1e-10 of
the largest attribution."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk

pytestmark = pytest.mark.gpu

KERNELS = {
    "t2": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 3}),
    "t4-l8": ("wgkm", {"L": 8, "k": 5, "d": 2}),
    "t2-l6": ("gkm_esttrunc", {"L": 6, "k": 4, "d": 2}),
}


@pytest.mark.parametrize("name", KERNELS)
@pytest.mark.parametrize("mode", ["importance", "hypothetical", "perturbation"])
def test_block_edges(name, mode):
    kt, params = KERNELS[name]
    l = params["L"]
    rng = np.random.default_rng(11)
    T = 128 - l + 1
    xl = np.array([T - 1, T, T + 1, 2 * T - 1, 2 * T, 2 * T + 1, 2 * T + l, l, l + 1])
    x = rng.integers(0, 4, (len(xl), xl.max() + 5)).astype(np.uint8)
    m = gk.GkmSVM(rng.integers(0, 4, (40, 60)).astype(np.uint8), rng.normal(size=40), 0.1, kt, params).cuda()
    out = []
    for use in (False, True):
        m.use_explain_table = use
        out.append(gk.gkmexplain(m, x, lengths=xl, mode=mode).cpu().numpy())
    np.testing.assert_allclose(out[1], out[0], rtol=0, atol=1e-10 * np.abs(out[0]).max())
