"""Ragged host batches tell the count tables' rule how many windows they have:
padding is not counted as work that the tables would save."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine
from gkmsvm_lite_b200.batch import DirectScorer
from gkmsvm_lite_b200.serve import GkmServer, GpuBackend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["predict", "ism", "explain", "variants", "impact", "direct", "serve"])
def test_windows(call, monkeypatch):
    rng = np.random.default_rng(12)
    m = gk.GkmSVM(syn.random_codes(rng, 100, 150), rng.normal(size=100), 0.1, "gkmrbf",
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    lengths = np.array([300, 40, 11, 60])
    x = syn.ragged_codes(rng, lengths)
    alt = (x + 1) % 4
    windows = int((lengths - 10).sum())
    asked, real = [], engine.DeviceIndex.table_bytes
    monkeypatch.setattr(engine.DeviceIndex, "table_bytes",
                        lambda self, B, W, windows=0: asked.append(windows) or real(self, B, W, windows))
    if call == "predict":
        m(x, lengths=lengths)
    elif call == "ism":
        gk.ism(m, x, lengths=lengths)
    elif call == "explain":
        gk.gkmexplain(m, x, lengths=lengths)
    elif call in ("variants", "impact"):
        windows *= 2
        m.score_variants(x, alt, ref_lengths=lengths, alt_lengths=lengths,
                         method="kernel" if call == "variants" else "gkmexplain")
    elif call == "direct":
        DirectScorer(m).score(torch.from_numpy(x).cuda(), torch.from_numpy(lengths).cuda(), windows=windows)
    else:
        with GkmServer(GpuBackend(m)) as server:
            server.submit("predict", x, lengths=lengths).result(60)
    assert asked == [windows]
