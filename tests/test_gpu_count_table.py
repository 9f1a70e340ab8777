"""Count-table queries (gkm_count_table_query) against the index walk: K_raw and
K(x, x) equal to the last bit (both weight the same exact integer counts in the
same order), scores within the rounding of two orders of the SV sum.  The sizes
are the edges: one row, a group of rows and one more, rows of no and of one
window, l = 8 .. 11 (odd l folds the strands into one table row), d = 0 .. 3, one
strand, low-complexity rows that overflow the shared counters and clip weighted
entries, and SV windows past them."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu

KERNELS = {
    "t3": ("gkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 2.0}),
    "t5": ("wgkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 1.0}),
    "t3-l10": ("gkmrbf", {"L": 10, "k": 6, "d": 3, "gamma": 1.0}),
    "t4-l10": ("wgkm", {"L": 10, "k": 6, "d": 3, "M": 20, "H": 10.0}),
    "t3-l9-d2": ("gkmrbf", {"L": 9, "k": 6, "d": 2, "gamma": 1.0}),
    "t4-l8-d1": ("wgkm", {"L": 8, "k": 5, "d": 1, "M": 5, "H": 20.0}),
    "t2-d0": ("gkm_esttrunc", {"L": 11, "k": 7, "d": 0}),
    "t3-one-strand": ("gkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 2.0, "include_rc": False}),
    "t5-one-strand": ("wgkmrbf", {"L": 10, "k": 6, "d": 3, "gamma": 1.0, "include_rc": False}),
}
# rows, shortest, longest, low-complexity rows among them
SHAPES = [(1, 64, 64, False), (32, 11, 40, False), (33, 100, 400, False), (5, 30, 700, True), (70, 200, 300, True)]


def _data(rng, n, lo, hi, low_complexity):
    xl = rng.integers(lo, hi + 1, n)
    xl[0] = hi
    x = syn.ragged_codes(rng, xl)
    if low_complexity:
        x[0] = 0  # poly-A
        xl[:4] = hi
        x[1] = np.tile([0, 3], hi)[:hi]  # its own reverse complement
        x[2, 20:60] = 2
        x[3] = np.tile([0, 1, 1], hi)[:hi]
    return x, xl


def _model(kt, params, rng, low_complexity, n_sv=150):
    sv, sl = _data(rng, n_sv, 20, 120, low_complexity)
    m = gk.GkmSVM(sv, rng.normal(size=n_sv), 0.3, kt, params, sv_lengths=sl).cuda()
    m.use_lmer_table = False
    return m


def _query(m, x, xl):
    spec = m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    index = m._sv_index()
    # more windows than there are: the walk then never looks cheaper
    n = index.table_bytes(*fwd.shape, 1 << 40)
    assert n > 0
    work = torch.full((n,), 0xAB, dtype=torch.uint8, device="cuda")
    return spec, fwd, rc, counts, index, work


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("name", KERNELS)
def test_equals_the_walk(name, shape):
    kt, params = KERNELS[name]
    B, lo, hi, low = shape
    rng = np.random.default_rng(B)
    m = _model(kt, params, rng, low)
    x, xl = _data(rng, B, lo, hi, low)
    if B > 6:
        xl[5], xl[6] = 0, params["L"]  # no window, one window
    spec, fwd, rc, counts, index, work = _query(m, x, xl)
    raw = torch.full((B, index.S), -1.0, dtype=torch.float64, device="cuda")
    diag = torch.empty(B, dtype=torch.float64, device="cuda")
    index.table_query(fwd, counts, work=work, raw=raw, diag=diag)
    want, _ = index.pairwise(fwd, counts)
    assert torch.equal(raw, want)
    dx = engine.self_kernel(spec, fwd, rc, counts)
    assert torch.equal(diag, dx)
    order = torch.argsort(counts, descending=True).to(torch.int32)
    scores = torch.empty(B, dtype=torch.float64, device="cuda")
    rbf, gamma = hasattr(m.kernel, "gamma"), getattr(m.kernel, "gamma", 0.0)
    index.table_query(fwd, counts, work=work, order=order, inv_ds=m._inv_ds(), coef=m._sv_coef(), gamma=gamma, rbf=rbf,
                      bias=0.3, scores=scores)
    inv_dx = 1.0 / torch.sqrt(torch.clamp(dx, min=1e-20))
    ref = index.score(fwd, counts, inv_dx, m._inv_ds(), m._sv_coef(), gamma, rbf, 0.3)
    np.testing.assert_allclose(scores.cpu().numpy(), ref.cpu().numpy(), rtol=1e-12, atol=1e-12)


def test_counts_of_the_oracle():
    """K_raw of a kernel whose pair weights are whole numbers (C(l - m, k)), where
    every sum is exact: the oracle's integer profiles weighted."""
    rng = np.random.default_rng(2)
    kt, params = "gkm_cnt_rbf", {"L": 11, "k": 7, "d": 3, "gamma": 1.0}
    m = _model(kt, params, rng, True)
    x, xl = _data(rng, 7, 100, 200, True)
    _, fwd, _, counts, index, work = _query(m, x, xl)
    raw = torch.empty((7, index.S), dtype=torch.float64, device="cuda")
    index.table_query(fwd, counts, work=work, raw=raw)
    prof = orc.profiles(x, xl, m.support_sequences, m.sv_lengths, orc.KernelDef.from_params(kt, params))
    h = m.kernel.base._mismatch_table[:4].astype(np.uint64)
    np.testing.assert_array_equal(raw.cpu().numpy(), (prof[..., :4] * h).sum(axis=-1).astype(np.float64))


@pytest.mark.parametrize("name", ["t3", "t5"])
def test_self_gram_writes_its_upper_triangle(name):
    kt, params = KERNELS[name]
    rng = np.random.default_rng(3)
    x, xl = _data(rng, 97, 30, 200, False)
    m = gk.GkmSVM(x, rng.normal(size=97), 0.0, kt, params, sv_lengths=xl).cuda()
    _, fwd, _, counts, index, work = _query(m, x, xl)
    raw = torch.full((97, 97), -1.0, dtype=torch.float64, device="cuda")
    index.table_query(fwd, counts, work=work, raw=raw, diag_offset=0)
    full, _ = index.pairwise(fwd, counts)
    upper = torch.triu(torch.ones_like(full)).bool()
    assert torch.equal(raw[upper], full[upper])
    assert bool((raw[~upper] == -1.0).all())


def test_refuses_what_it_cannot_hold():
    """A workspace too small or misaligned, both outputs at once and a count
    that could reach 2^32 are refused (the last goes to the walk)."""
    kt, params = KERNELS["t3"]
    rng = np.random.default_rng(4)
    m = _model(kt, params, rng, False)
    x, xl = _data(rng, 2, 50, 60, False)
    _, fwd, _, counts, index, work = _query(m, x, xl)
    raw = torch.empty((2, index.S), dtype=torch.float64, device="cuda")
    for bad in (work[:-256], work[1:]):
        with pytest.raises(gk._lib.GkmError):
            index.table_query(fwd, counts, work=bad, raw=raw)
    with pytest.raises(ValueError):
        index.table_query(fwd, counts, work=work, raw=raw, scores=raw[:, 0], inv_ds=raw[0], coef=raw[0])
    heavy = _model("wgkmrbf", {"L": 11, "k": 7, "d": 3, "gamma": 1.0, "M": 255, "H": 1e6}, rng, False)
    assert heavy._sv_index().table_bytes(2, 50, 1 << 40) == 0
    assert index.table_bytes(2, 50000, 1 << 40) == 0
