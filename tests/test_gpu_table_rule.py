"""Which shapes the count tables' rule sends to them: those measured faster so, and
not short l-mers whose few tiles list or recount most windows."""

import numpy as np
import pytest

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn

pytestmark = pytest.mark.gpu


# SVs, weighted, l, d, rows, length; milliseconds of the walk and of the tables
@pytest.mark.parametrize("shape,walk,tables", [
    ((64, 1, 8, 2, 1024, 2000), 5.3, 61.7), ((500, 0, 8, 2, 1024, 300), 1.5, 3.4), ((500, 1, 8, 3, 1024, 30), 1.1, 3.4),
    ((64, 1, 9, 3, 1024, 100), 1.9, 4.0), ((64, 1, 8, 1, 256, 1000), 0.66, 0.89), ((3000, 0, 11, 3, 64, 300), 1.67, 0.33),
    ((3000, 1, 10, 3, 64, 300), 1.36, 0.47), ((500, 0, 8, 1, 1, 300), 0.53, 0.04), ((500, 0, 9, 3, 16, 300), 0.73, 0.08)])
def test_faster_form(shape, walk, tables):
    S, weighted, l, d, B, L = shape
    rng = np.random.default_rng(0)
    lengths = rng.integers(200, 351, S)
    m = gk.GkmSVM(syn.ragged_codes(rng, lengths), rng.normal(size=S), 0.1, "wgkmrbf" if weighted else "gkmrbf",
                  {"L": l, "k": l - 4, "d": d, "gamma": 1.0}, sv_lengths=lengths).cuda()
    W = L - l + 1
    assert (m._sv_index().table_bytes(B, W, B * W) > 0) == (tables < walk)
