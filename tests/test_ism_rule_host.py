"""ISM's choice between pair lists and the index walk at shapes measured in both
forms (B200; SVs of 200 .. 350 bp)."""

import types

import numpy as np
import pytest
import torch

from gkmsvm_lite_b200 import kernels as K
from gkmsvm_lite_b200.ism import _pairs_pay


# SVs, index entries, tiles, weighted, l, d, rows, length; microseconds of pair lists and walk
@pytest.mark.parametrize("S,entries,tiles,weighted,l,d,B,L,pairs,walk", [
    (64, 33332, 1, 0, 11, 3, 1, 400, 143, 598),
    (64, 33332, 1, 0, 11, 3, 64, 20, 2605, 1034),
    (64, 33332, 1, 0, 11, 1, 64, 60, 2377, 512),
    (64, 33332, 1, 0, 11, 1, 4, 1000, 252, 540),
    (64, 33716, 1, 1, 8, 3, 16, 150, 1759, 879),
    (3000, 1592358, 1, 0, 11, 3, 16, 150, 1739, 3979),
    (3000, 1610358, 1, 0, 8, 1, 64, 60, 3970, 1252),
    (3000, 1610358, 1, 0, 8, 1, 1, 1000, 178, 375),
    (72000, 38161654, 2, 0, 11, 3, 1, 400, 1625, 3410),
    (72000, 38161654, 6, 1, 11, 3, 1, 1000, 3804, 12657),
    (72000, 38161654, 2, 0, 11, 3, 16, 20, 9337, 2119),
    (72000, 38161654, 2, 0, 11, 1, 64, 60, 34408, 18820),
    (72000, 38593654, 6, 1, 8, 3, 4, 400, 40313, 79121)])
def test_faster_form(S, entries, tiles, weighted, l, d, B, L, pairs, walk):
    base = (K.CenterWeightedGkmKernel if weighted else K.EstTruncGkmKernel)(l, l - 4, d=d)
    index = types.SimpleNamespace(S=S, entries=entries, tiles=tiles,
                                  masks=torch.zeros(K.neighbor_count(l, d), dtype=torch.int32))
    assert _pairs_pay(base, index, B, L, 148) == (pairs < walk)


def test_one_strand_and_short_rows():
    """Every shape the entry points take has an answer."""
    for l, d, L in ((8, 0, 8), (11, 3, 11), (11, 3, 2048)):
        base = K.EstTruncGkmKernel(l, l - 4, d=d, include_rc=False)
        index = types.SimpleNamespace(S=64, entries=1, tiles=1, masks=np.empty(0))
        index.masks = torch.zeros(K.neighbor_count(l, d), dtype=torch.int32)
        assert _pairs_pay(base, index, 1, L, 148) in (True, False)
