"""K(x, x) by bit-sliced diagonals (gkm_self_kernel): profiles equal to the
oracle's at the edges of the 32-pair words (rows of 1 window, of 31..33, of 63..65,
ragged), every template (l = 10, 11 and the run-time length, up to 4 levels and
more, weighted, one strand), low-complexity rows, and rows whose windows are not
one sequence's (taken pair by pair)."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu

KERNELS = {
    "t2": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 3}),
    "t4": ("wgkm", {"L": 11, "k": 7, "d": 3}),
    "t2-l10": ("gkm_esttrunc", {"L": 10, "k": 6, "d": 3}),
    "t4-l10": ("wgkm", {"L": 10, "k": 6, "d": 2}),
    "t0-l6": ("gkm_cnt", {"L": 6, "k": 4}),
    "t0-l11": ("gkm_cnt", {"L": 11, "k": 7}),
    "t0-l15": ("gkm_cnt", {"L": 15, "k": 6, "d": 9}),
    "t4-l7-d5": ("wgkm", {"L": 7, "k": 2, "d": 5, "M": 255, "H": 9.0}),
    "t2-one-strand": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 3, "include_rc": False}),
}


@pytest.mark.parametrize("name", KERNELS)
def test_profiles_of_the_oracle(name):
    kt, params = KERNELS[name]
    rng = np.random.default_rng(5)
    l = params["L"]
    xl = np.array([l, l + 1, l + 30, l + 31, l + 32, l + 62, l + 63, l + 64, 200, 333, 120, 90])
    x = rng.integers(0, 4, (len(xl), xl.max())).astype(np.uint8)
    x[-2] = 0
    x[-1] = np.tile([0, 3], xl.max())[: xl.max()]
    kd = orc.KernelDef.from_params(kt, params)
    m = gk.GkmSVM(x[:2], np.ones(2), 0.0, kt, params).cuda()
    spec = m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    _, prof = engine.self_kernel(spec, fwd, rc, counts, profile=True)
    want = orc.self_profiles(x, xl, kd)
    d = kd.dmax
    np.testing.assert_array_equal(prof.cpu().numpy()[:, : d + 1].astype(np.uint64), want[:, : d + 1])


@pytest.mark.parametrize("name", ["t2", "t4"])
def test_windows_of_no_one_sequence(name):
    """Packed windows in reverse order have the K(x, x) of the row in sequence
    order; they overlap no more, so they are taken pair by pair."""
    kt, params = KERNELS[name]
    rng = np.random.default_rng(6)
    x = rng.integers(0, 4, (3, 150)).astype(np.uint8)
    m = gk.GkmSVM(x, np.ones(3), 0.0, kt, params).cuda()
    spec = m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), None)
    flip = lambda t: torch.flip(t, [1]).contiguous()
    # 139 windows: the window weights are symmetric about the centre
    fwd, rc = fwd[:, :139].contiguous(), rc[:, -139:].contiguous()
    counts = torch.full_like(counts, 139)
    _, want = engine.self_kernel(spec, fwd, rc, counts, profile=True)
    _, got = engine.self_kernel(spec, flip(fwd), flip(rc), counts, profile=True)
    assert torch.equal(got, want)
