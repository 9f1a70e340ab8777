"""RBF attributions by l-mer weights per row and by the buckets, each forced: the
same within the rounding of sums in other orders (1e-12 of the largest attribution,
a few thousand terms); more rows than one buffer of weights holds; and the buckets
where the device has no room for the weights."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import explain

pytestmark = pytest.mark.gpu


def _model(kt, l, d, n_sv=200):
    rng = np.random.default_rng(l)
    sl = rng.integers(20, 150, n_sv)
    return gk.GkmSVM(syn.ragged_codes(rng, sl), rng.normal(size=n_sv), 0.0, kt, {"L": l, "k": l - 4, "d": d, "gamma": 1.0},
                     sv_lengths=sl).cuda()


@pytest.mark.parametrize("mode", ["hypothetical", "perturbation"])
@pytest.mark.parametrize("rows", [1, 7, 18])
@pytest.mark.parametrize("kt,l,d", [("gkmrbf", 6, 2), ("wgkmrbf", 8, 1), ("gkmrbf", 11, 2), ("wgkmrbf", 12, 2)])
def test_forms_agree(kt, l, d, rows, mode, monkeypatch):
    m = _model(kt, l, d)
    rng = np.random.default_rng(rows)
    xl = rng.integers(l, 80, rows)
    xl[0] = 80
    x = syn.ragged_codes(rng, xl)
    called, real, got = [], explain.call, {}
    monkeypatch.setattr(explain, "call", lambda name, *a: called.append(name) or real(name, *a))
    for pay in (True, False):
        monkeypatch.setattr(explain, "_row_weights_pay", lambda *a: pay)
        got[pay] = gk.gkmexplain(m, x, lengths=xl, mode=mode).cpu().numpy()
    assert "gkm_explain_subsets" in called and called.count("gkm_explain_lmer") == 1
    np.testing.assert_allclose(got[True], got[False], rtol=0, atol=1e-12 * np.abs(got[False]).max())


def test_no_room_for_the_weights(monkeypatch):
    m = _model("gkmrbf", 11, 3)
    x = syn.random_codes(np.random.default_rng(1), 8, 60)
    monkeypatch.setattr(explain, "_row_weights_pay", lambda *a: True)
    want = gk.gkmexplain(m, x).cpu().numpy()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    called, real = [], explain.call
    monkeypatch.setattr(explain, "call", lambda name, *a: called.append(name) or real(name, *a))
    total = torch.cuda.mem_get_info()[1]
    try:  # 8 rows of weights take 268 MB
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (200 << 20)) / total)
        got = gk.gkmexplain(m, x).cpu().numpy()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert "gkm_explain_lmer" in called
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())
