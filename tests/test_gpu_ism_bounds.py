"""gkm_ism_pairs serves rows whose windows lie within the positions it writes and
refuses others."""

import ctypes

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200._lib import call, ptr, stream_handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [64, 512, 1024, 2048])
def test_windows_past_the_positions(L):
    rng = np.random.default_rng(7)
    m = gk.GkmSVM(syn.random_codes(rng, 100, 200), rng.normal(size=100), 0.1, "gkmrbf",
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    index = m._sv_index()
    n = ctypes.c_int64()
    call("gkm_ism_pairs_workspace", index.handle, L - 10, L, ctypes.byref(n))
    assert n.value > 0
    work = torch.empty(n.value + (1 << 24), dtype=torch.uint8, device="cuda")
    for W in (L - 9, L):
        call("gkm_ism_pairs_workspace", index.handle, W, L, ctypes.byref(n))
        assert n.value == 0
        fwd = torch.zeros((1, W), dtype=torch.int32, device="cuda")
        counts = torch.full((1,), W, dtype=torch.int32, device="cuda")
        raw = torch.zeros((1, index.S), dtype=torch.float64, device="cuda")
        one = torch.ones(1, dtype=torch.float64, device="cuda")
        mut = torch.ones((4, L, 1), dtype=torch.float64, device="cuda")
        out = torch.full((1, 4, L), -1.0, dtype=torch.float64, device="cuda")
        with pytest.raises(gk._lib.GkmError):
            call("gkm_ism_pairs", index.handle, ptr(fwd), ptr(counts), 1, W, L, ptr(raw), ptr(one), ptr(mut),
                 ptr(m._inv_ds()), ptr(m._sv_coef()), 1.0, 1, ptr(out), ptr(work), int(work.numel()), stream_handle())
        assert bool((out == -1.0).all())
