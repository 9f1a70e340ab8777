"""ISM by pair lists and by the index walk, each forced, at the shapes where the
rule between them can go either way: the same deltas within the rounding of sums
over the SVs in another order (1e-12 of the largest score)."""

import importlib

import numpy as np
import pytest

import gkmsvm_lite_b200 as gk

ism_module = importlib.import_module("gkmsvm_lite_b200.ism")  # (the package's ism is the function)
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,l,d", [("gkmrbf", 11, 3), ("wgkmrbf", 11, 1), ("gkmrbf", 8, 1), ("wgkmrbf", 8, 3),
                                    ("gkmrbf", 10, 2), ("wgkmrbf", 9, 0)])
@pytest.mark.parametrize("B,L", [(1, 300), (9, 40), (3, 600)])
def test_forms_agree(kt, l, d, B, L, monkeypatch):
    rng = np.random.default_rng(B * L)
    S = 300
    sl = rng.integers(20, 200, S)
    sv = rng.integers(0, 4, (S, 200)).astype(np.uint8)
    m = gk.GkmSVM(sv, rng.normal(size=S), 0.3, kt, {"L": l, "k": l - 4, "d": d, "gamma": 1.0}, sv_lengths=sl).cuda()
    x = rng.integers(0, 4, (B, L)).astype(np.uint8)
    xl = rng.integers(l, L + 1, B)
    xl[0] = L
    called, real, got = [], ism_module.call, {}
    monkeypatch.setattr(ism_module, "call", lambda name, *a: called.append(name) or real(name, *a))
    for pairs in (True, False):
        monkeypatch.setattr(ism_module, "_pairs_pay", lambda *a: pairs)
        got[pairs] = gk.ism(m, x, lengths=xl).cpu().numpy()
    assert called.count("gkm_ism_pairs") == 1 and called.count("gkm_index_mutants") == 1
    scale = float(m(x, lengths=xl).abs().max()) + float(np.abs(got[False]).max())
    np.testing.assert_allclose(got[True], got[False], rtol=0, atol=1e-12 * scale)
