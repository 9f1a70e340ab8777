"""Weighted K(x, x) by diagonals and pair by pair, on both sides of the rule between
them: profiles equal to the oracle's."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import _lib, engine

pytestmark = pytest.mark.gpu

FORMS = ["diagonals", "pairs"]


# l, d, rows, longest row, form
@pytest.mark.parametrize("l,d,B,L,form", [
    (7, 5, 12, 300, "pairs"), (7, 5, 320, 110, "diagonals"), (9, 5, 3, 600, "pairs"), (9, 4, 3, 600, "diagonals"),
    (4, 3, 3, 300, "pairs"), (6, 2, 3, 300, "diagonals"), (12, 10, 4, 300, "pairs"), (13, 8, 4, 300, "diagonals")])
@pytest.mark.parametrize("strands", [1, 2])
def test_profiles_of_the_oracle(l, d, B, L, form, strands):
    params = {"L": l, "k": l - d, "d": d, "M": 255, "H": 30.0, "include_rc": strands == 2}
    rng = np.random.default_rng(l)
    xl = rng.integers(l, L + 1, B)
    xl[0], xl[1], xl[-1] = L, l, 0
    x = rng.integers(0, 4, (B, L)).astype(np.uint8)
    x[2] = np.tile([0, 3], L)[:L]
    kd = orc.KernelDef.from_params("wgkm", params)
    m = gk.GkmSVM(x[:2], np.ones(2), 0.0, "wgkm", params).cuda()
    assert m.kernel.base.dmax == d
    spec = m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    assert FORMS[_lib.load().gkm_self_form(spec.ref, *fwd.shape)] == form
    _, prof = engine.self_kernel(spec, fwd, rc, counts, profile=True)
    rows = [0, 1, 2, B - 2]
    want = orc.self_profiles(x[rows], xl[rows], kd)
    np.testing.assert_array_equal(prof.cpu().numpy()[rows, : d + 1].astype(np.uint64), want[:, : d + 1])
    assert int(prof[B - 1].sum()) == 0
