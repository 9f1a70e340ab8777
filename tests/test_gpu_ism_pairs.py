"""ISM deltas from pair lists (gkm_ism_pairs) against the index walk
(gkm_index_mutants): the same deltas within the rounding of sums over the SVs taken
in another order (1e-12 of the largest score).  The sizes are the edges: rows of one
window and of none, positions past 512 and 1,024 (wider blocks), l = 8 .. 11, d = 0 ..
3, one strand, weighted, linear, low-complexity rows and SVs, one SV more than a
multiple of the grid's small cases."""

import ctypes

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import engine
from gkmsvm_lite_b200._lib import call
from gkmsvm_lite_b200.ism import _ism_index, ism_pass_bytes, ism_workspace

pytestmark = pytest.mark.gpu

KERNELS = {
    "t3": ("gkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 2.0}),
    "t5": ("wgkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 1.0}),
    "t5-heavy": ("wgkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 1.0, "M": 85, "H": 100.0}),
    "t3-l10": ("gkmrbf", {"L": 10, "k": 6, "d": 3, "gamma": 1.0}),
    "t3-l9-d2": ("gkmrbf", {"L": 9, "k": 6, "d": 2, "gamma": 1.0}),
    "t4-l8-d1": ("wgkm", {"L": 8, "k": 5, "d": 1}),
    "t2-d0": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 0}),
    "t3-one-strand": ("gkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 2.0, "include_rc": False}),
    "t5-l10-one-strand": ("wgkmrbf", {"L": 10, "k": 6, "d": 3, "gamma": 1.0, "include_rc": False}),
}


def _model(rng, kt, params, S):
    sl = rng.integers(20, 200, S)
    sv = rng.integers(0, 4, (S, 200)).astype(np.uint8)
    sv[0], sl[0] = 0, 200
    sv[1, 5:18] = 3
    m = gk.GkmSVM(sv, rng.normal(size=S), 0.3, kt, params, sv_lengths=sl).cuda()
    m.use_lmer_table = False
    return m


@pytest.mark.parametrize("name", KERNELS)
@pytest.mark.parametrize("L", [64, 513, 1030])
def test_equals_the_walk(name, L):
    kt, params = KERNELS[name]
    l = params["L"]
    rng = np.random.default_rng(L)
    m = _model(rng, kt, params, 65)
    xl = np.array([L, l, l + 1, L - 1])
    x = rng.integers(0, 4, (4, L)).astype(np.uint8)
    x[3, 10:40] = 0
    spec, index = m._spec(), m._sv_index()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    counts[1] = 0  # a padding row
    n = ctypes.c_int64()
    call("gkm_ism_pairs_workspace", index.handle, fwd.shape[1], L, ctypes.byref(n))
    assert n.value > 0
    got = _ism_index(m, fwd, rc, counts, L)
    small = ism_workspace(m, 4, L, fwd.device, cap=ism_pass_bytes(m, 4, 8))
    assert small.numel() < n.value  # too small for the lists: the walk
    want = _ism_index(m, fwd, rc, counts, L, work=small)
    assert torch.equal(got[1], torch.zeros_like(got[1]))
    scale = float(m(x, lengths=xl).abs().max()) + float(want.abs().max())
    np.testing.assert_allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=0, atol=1e-12 * scale)


def test_long_rows_take_the_walk():
    rng = np.random.default_rng(0)
    m = _model(rng, "gkmrbf", {"L": 11, "k": 7, "d": 3}, 65)
    n = ctypes.c_int64(-1)
    call("gkm_ism_pairs_workspace", m._sv_index().handle, 2039, 2049, ctypes.byref(n))
    assert n.value == 0
