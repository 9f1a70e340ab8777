"""gkm_count_table_query refuses a shape whose counts could wrap, whatever
workspace it is given."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu


def test_counts_that_could_pass_32_bits():
    rng = np.random.default_rng(6)
    # every window weighs 80: 80 * 20,000 of the row times 80 * 190 of an SV, both strands
    m = gk.GkmSVM(syn.random_codes(rng, 100, 200), rng.normal(size=100), 0.1, "wgkmrbf",
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0, "M": 80, "H": 1e9}).cuda()
    index = m._sv_index()
    x = torch.from_numpy(syn.random_codes(rng, 1, 20_010)).cuda()
    fwd, _, counts = engine.pack(m._spec(), x, None)
    assert index.table_bytes(*fwd.shape, 1 << 40) == 0
    assert index.table_bytes(1, 200, 1 << 40) > 0  # (the index has count tables)
    work = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
    raw = torch.full((1, index.S), -1.0, dtype=torch.float64, device="cuda")
    with pytest.raises(gk._lib.GkmError, match="2\\^32"):
        index.table_query(fwd, counts, work=work, raw=raw)
    assert bool((raw == -1.0).all())
