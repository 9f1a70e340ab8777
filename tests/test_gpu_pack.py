"""Packed windows at the edges of a packing block (1,024 windows) and of rows with blocks
of their own (256 windows): rows of no, one,
1,023 .. 1,025 and 2,049 windows, rows shorter than the batch, without lengths, l =
2, 8, 11, 15, rows at odd byte offsets.  Exact."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l", [2, 8, 11, 15])
@pytest.mark.parametrize("W", [1, 3, 255, 256, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("ragged", [False, True])
def test_windows(l, W, ragged):
    L = W + l - 1
    rng = np.random.default_rng(W + l)
    x = rng.integers(0, 4, (5, L)).astype(np.uint8)
    xl = np.array([L, l - 1, l, max(l, L - 1), max(l, L // 2)]) if ragged else None
    spec = engine.Spec(gk.EstTruncGkmKernel(l, min(l, 6), d=1), torch.device("cuda"))
    fwd, rc, counts = (t.cpu().numpy().astype(np.int64) & 0xFFFFFFFF for t in
                       engine.pack(spec, torch.from_numpy(x).cuda(), xl))
    n = np.clip((xl if ragged else np.full(5, L)) - l + 1, 0, W)
    np.testing.assert_array_equal(counts, n)
    for b in range(5):
        want = np.full(W, 0xFFFFFFFF, np.int64)
        want_rc = want.copy()
        for i in range(n[b]):
            w = x[b, i : i + l].astype(np.int64)
            want[i] = (w << (2 * np.arange(l))).sum()
            want_rc[W - 1 - i] = ((3 - w[::-1]) << (2 * np.arange(l))).sum()
        np.testing.assert_array_equal(fwd[b], want)
        np.testing.assert_array_equal(rc[b], want_rc)
