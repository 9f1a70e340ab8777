"""GkmExplain by position subsets (gkm_explain_subsets) against gkm_explain_lmer's
per-mask loop on the same l-mer weights, and row_weights against their definition:
2 to 4 mismatches, importance and perturbation tables, weighted windows, ragged
rows, one row to more than four, weights per row and shared.  The two add the same
terms in other orders; the largest sum has ~3,400 terms, so 1e-12 of the largest
attribution is ~1.4 times the worst rounding of either."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine, explain
from gkmsvm_lite_b200._lib import call, ptr, stream_handle

pytestmark = pytest.mark.gpu

KERNELS = {
    "t2": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 3}),
    "t4-l10": ("wgkm", {"L": 10, "k": 6, "d": 2}),
    "t3-l9": ("gkmrbf", {"L": 9, "k": 6, "d": 3, "gamma": 1.0}),
    "t5-l12": ("wgkmrbf", {"L": 12, "k": 8, "d": 2, "gamma": 1.0}),
    "t3-one-strand": ("gkmrbf", {"L": 9, "k": 6, "d": 3, "gamma": 1.0, "include_rc": False}),
}


@pytest.mark.parametrize("perturbation", [False, True])
@pytest.mark.parametrize("rows", [1, 5])
@pytest.mark.parametrize("name", KERNELS)
def test_equals_the_mask_loop(name, rows, perturbation):
    kt, params = KERNELS[name]
    rng = np.random.default_rng(rows)
    sl = rng.integers(20, 150, 200)
    m = gk.GkmSVM(syn.ragged_codes(rng, sl), rng.normal(size=200), 0.0, kt, params, sv_lengths=sl).cuda()
    dev = m._require_gpu()
    spec, index = m._spec(), m._sv_index()
    xl = rng.integers(params["L"], 90, rows)
    xl[0] = 90
    x = syn.ragged_codes(rng, xl)
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    (B, W), L, l = fwd.shape, x.shape[1], params["L"]
    inv_dx = torch.rand(B, dtype=torch.float64, device=dev)
    w = torch.randn((B, index.S), dtype=torch.float64, device=dev)
    masks, ta, tb = explain._explain_masks(m, perturbation, dev)
    subs, lists, n_with, size = explain._explain_subsets(m, perturbation, dev)
    V = torch.empty((B, 4**l), dtype=torch.float64, device=dev)
    for g in range(0, B, 4):
        k = min(4, B - g)
        width = {1: 2, 4: 4}[k]
        ws = torch.full((index.S, width), 7.0, dtype=torch.float64, device=dev)
        ws[:, :k] = w[g:g + k].T
        call("gkm_index_row_weights", index.handle, ptr(ws), width, k, ptr(V[g]), stream_handle())
    for r in range(B):
        want = index.lmer_weights(w[r].contiguous())
        torch.testing.assert_close(V[r], want, rtol=1e-12, atol=1e-12 * float(want.abs().max()))
    part = torch.full((B, W, 4, l), np.nan, dtype=torch.float64, device=dev)
    for per_row in (True, False):
        got = torch.full((B, 4, L), np.nan, dtype=torch.float64, device=dev)
        call("gkm_explain_subsets", spec.ref, ptr(fwd), ptr(counts), B, W, L, ptr(inv_dx), ptr(V), 4**l if per_row else 0,
             ptr(subs), int(subs.numel()), size, ptr(lists), ptr(n_with), ptr(ta), ptr(tb), int(perturbation), ptr(part),
             ptr(got), stream_handle())
        want = torch.empty_like(got)
        call("gkm_explain_lmer", spec.ref, ptr(fwd), ptr(counts), B, W, L, ptr(inv_dx), None if per_row else ptr(V),
             index.handle if per_row else None, ptr(w) if per_row else None, ptr(masks), int(masks.numel()), ptr(ta),
             ptr(tb), int(perturbation), ptr(want), stream_handle())
        torch.testing.assert_close(got, want, rtol=0, atol=1e-12 * float(want.abs().max()))
