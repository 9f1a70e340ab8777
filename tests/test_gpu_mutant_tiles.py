"""Mutant self-kernels by bit-sliced diagonals (gkm_mutant_diag) against the
self-kernels of the substituted rows, at the edges of the position tiles (128 -
2 (l - 1) and 128 - l + 1 positions), rows of one window, ragged and low-complexity
rows, l = 8 (run-time length), 10, 11, one strand, weighted windows, d = 1 .. 3 and
(the pair loop) 4 levels and more.  Both weight exact integer counts: the mutant's is
K(x, x) plus four products, a handful of roundings of values near K(x, x), so 1e-12."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu

KERNELS = {
    "t2": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 3}),
    "t4": ("wgkm", {"L": 11, "k": 7, "d": 3}),
    "t2-l10-d2": ("gkm_esttrunc", {"L": 10, "k": 6, "d": 2}),
    "t4-l8-d1": ("wgkm", {"L": 8, "k": 5, "d": 1, "M": 255, "H": 4.0}),
    "t2-one-strand": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 3, "include_rc": False}),
    "t0-l6": ("gkm_cnt", {"L": 6, "k": 2}),
}


@pytest.mark.parametrize("name", KERNELS)
def test_equals_the_substituted_rows(name):
    kt, params = KERNELS[name]
    l = params["L"]
    rng = np.random.default_rng(8)
    xl = np.array([l, l + 1, 128 - l, 128, 129, 128 + l, 300, 150, 90])
    x = rng.integers(0, 4, (len(xl), xl.max())).astype(np.uint8)
    x[-2] = np.tile([0, 3], xl.max())[: xl.max()]
    x[-1, 20:60] = 1
    L = x.shape[1]
    m = gk.GkmSVM(x[:2], np.ones(2), 0.0, kt, params).cuda()
    spec = m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    diag = engine.self_kernel(spec, fwd, rc, counts)
    got = engine.mutant_diag(spec, fwd, counts, L, diag).cpu().numpy()  # [4, L, B]
    for b, n in enumerate(xl):
        mut = np.repeat(x[b : b + 1], 4 * n, axis=0)
        mut[np.arange(4 * n), np.arange(4 * n) % n] = np.arange(4 * n) // n
        f, r, c = engine.pack(spec, torch.from_numpy(mut).cuda(), np.full(4 * n, n))
        want = engine.self_kernel(spec, f, r, c).cpu().numpy().reshape(4, n)
        np.testing.assert_allclose(got[:, :n, b], want, rtol=1e-12)
        np.testing.assert_array_equal(got[:, n:, b], float(diag[b]))
