"""A warmed server holds one workspace per scorer, not one per bucket."""

import numpy as np
import pytest

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200.engine import DeviceIndex
from gkmsvm_lite_b200.serve import GpuBackend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", ["gkmrbf", "wgkmrbf"])
def test_warm_makes_one_workspace(kt):
    rng = np.random.default_rng(3)
    m = gk.GkmSVM(syn.random_codes(rng, 300, 200), rng.normal(size=300), 0.1, kt,
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    index = m._sv_index()
    index.table_bytes = lambda B, W, windows=0: DeviceIndex.table_bytes(index, B, W, 1 << 40)  # tables for every shape
    index.tables_pay = lambda *a: True
    backend = GpuBackend(m)
    backend.warm(max_len=512, max_rows=3072)
    for scorer in backend.scorers:
        assert len(scorer._graphs) == 3 * 4
        assert len(scorer.work._buffers) == 1
    assert all(len(r.table_work._buffers) <= 2 for r in backend.side_runners.values())
