"""ISM by pair lists and by the index walk, each forced, at the shapes where the
rule between them can go either way: the same deltas within the rounding of sums
over the SVs in another order (1e-12 of the largest score)."""

import importlib

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200.batch import BatchedIsm

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


@pytest.mark.parametrize("kt", ["gkmrbf", "wgkmrbf"])
def test_short_passes_take_the_form_of_the_call(kt, monkeypatch):
    """A runner's limit on the positions of a walk's pass leaves the choice of the
    form as it is: 8 rows of 512 positions against 300 SVs, 128 positions a pass."""
    rng = np.random.default_rng(3)
    sv = rng.integers(0, 4, (300, 200)).astype(np.uint8)
    m = gk.GkmSVM(sv, rng.normal(size=300), 0.3, kt, {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    x = rng.integers(0, 4, (8, 512)).astype(np.uint8)
    called, real = [], ism_module.call
    monkeypatch.setattr(ism_module, "call", lambda name, *a: called.append(name) or real(name, *a))
    want = gk.ism(m, x).cpu().numpy()
    scale = float(m(x).abs().max()) + float(np.abs(want).max())
    runner = BatchedIsm(m, pass_positions=128)
    for _ in range(3):  # eager, captured, replayed
        got = runner(torch.from_numpy(x).cuda()).cpu().numpy()
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * scale)
    assert called.count("gkm_ism_pairs") >= 2 and "gkm_index_mutants" not in called
