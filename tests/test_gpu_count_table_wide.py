"""Count tables of dense unweighted rows (four bytes per query) and gathers whose lane
groups share an SV, against the index walk: K_raw and K(x, x) bit for bit (whole counts
times the same weights in the same order).  l = 10 and 11 on both sides of the mean
count where entries widen, rows with and without low-complexity stretches (counts past
a byte, tiles counted again), one row and more than a group, S = 64 .. 3,000 (every
power of two of lane groups), weighted and not."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu


def _model(rng, kt, l, S, poly):
    sl = rng.integers(60, 200, S)
    sv = rng.integers(0, 4, (S, 200)).astype(np.uint8)
    if poly:
        sv[0], sl[0] = 0, 200
        sv[1, 5:40] = 0
    m = gk.GkmSVM(sv, rng.normal(size=S), 0.0, kt, {"L": l, "k": 6, "d": 3}, sv_lengths=sl).cuda()
    m.use_lmer_table = False
    return m


def _compare(m, x, xl, windows):
    index, spec = m._sv_index(), m._spec()
    fwd, rc, counts = engine.pack(spec, torch.from_numpy(x).cuda(), xl)
    B = len(xl)
    n = max(index.table_bytes(*fwd.shape, 1 << 40), index.table_bytes(*fwd.shape, windows))
    assert n > 0
    raw = torch.full((B, index.S), -1.0, dtype=torch.float64, device="cuda")
    diag = torch.empty(B, dtype=torch.float64, device="cuda")
    work = torch.full((n,), 0xAB, dtype=torch.uint8, device="cuda")
    index.table_query(fwd, counts, work=work, raw=raw, diag=diag, windows=windows)
    want, _ = index.pairwise(fwd, counts)
    assert torch.equal(raw, want)
    assert torch.equal(diag, engine.self_kernel(spec, fwd, rc, counts))


@pytest.mark.parametrize("l,n", [(10, 400), (10, 700), (10, 900), (11, 1200), (11, 2400)])
@pytest.mark.parametrize("poly", [False, True])
def test_dense_rows(l, n, poly):
    rng = np.random.default_rng(n)
    m = _model(rng, "gkmrbf", l, 300, poly)
    for B in (1, 33):
        xl = rng.integers(n // 2, n + 1, B)
        xl[0] = n
        x = rng.integers(0, 4, (B, n)).astype(np.uint8)
        if poly:
            x[0, 100:300] = 0
            x[-1, :60] = np.tile([0, 3], 30)
        for windows in (0, int((xl - l + 1).sum())):
            _compare(m, x, xl, windows)


@pytest.mark.parametrize("kt", ["gkmrbf", "wgkmrbf"])
@pytest.mark.parametrize("S", [64, 130, 700, 1500, 3000])
def test_few_svs(kt, S):
    rng = np.random.default_rng(S)
    m = _model(rng, kt, 11, S, True)
    for B in (3, 20, 40):
        xl = rng.integers(11, 121, B)
        x = rng.integers(0, 4, (B, 120)).astype(np.uint8)
        x[0] = 0
        _compare(m, x, xl, 1 << 40)
