"""Mutant self-kernels of a batch (mutant_tiles: by bit-sliced diagonals) and of its
rows one by one (mutant_kernel: a block per position), on both sides of the rule
between them: equal to the last bit, because both weight the same integer counts in
one order."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import _lib, engine

pytestmark = pytest.mark.gpu

FORMS = ["mutant_kernel", "mutant_tiles"]


# kernel type, l, d, rows, length; the forms of the batch and of one row
@pytest.mark.parametrize("kt,l,d,B,L,batch,row", [
    ("gkm_esttrunc", 11, 3, 64, 300, "mutant_tiles", "mutant_kernel"),
    ("wgkm", 11, 3, 64, 300, "mutant_tiles", "mutant_kernel"),
    ("gkm_esttrunc", 10, 2, 200, 150, "mutant_tiles", "mutant_kernel"),
    ("wgkm", 8, 1, 64, 200, "mutant_tiles", "mutant_kernel"),
    ("gkm_cnt", 6, 3, 32, 300, "mutant_kernel", "mutant_kernel"),
    ("wgkm", 6, 2, 16, 300, "mutant_kernel", "mutant_kernel"),
    ("gkm_esttrunc", 11, 3, 2, 2047, "mutant_tiles", "mutant_tiles")])
def test_forms_agree(kt, l, d, B, L, batch, row):
    rng = np.random.default_rng(B)
    xl = rng.integers(l, L + 1, B)
    xl[0] = L
    x = rng.integers(0, 4, (B, L)).astype(np.uint8)
    x[-1] = np.tile([0, 3], L)[:L]
    m = gk.GkmSVM(x[:2], np.ones(2), 0.0, kt, {"L": l, "k": l - d if kt == "gkm_cnt" else 4, "d": d}).cuda()
    assert m.kernel.base.dmax == d
    spec = m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    diag = engine.self_kernel(spec, fwd, rc, counts)
    W, form = fwd.shape[1], _lib.load().gkm_mutant_form
    assert (FORMS[form(spec.ref, B, W, L)], FORMS[form(spec.ref, 1, W, L)]) == (batch, row)
    got = engine.mutant_diag(spec, fwd, counts, L, diag)
    for b in range(0, B, max(1, B // 8)):
        one = engine.mutant_diag(spec, fwd[b:b + 1].contiguous(), counts[b:b + 1].contiguous(), L,
                                 diag[b:b + 1].contiguous())
        assert torch.equal(one[:, :, 0], got[:, :, b])
