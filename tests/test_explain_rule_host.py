"""GkmExplain's choice between l-mer weights per row and the buckets of the windows'
neighbourhoods, at RBF shapes measured in both forms (B200; SVs of 200 .. 350 bp)."""

import types

import pytest

from gkmsvm_lite_b200 import explain


# SVs, index entries, l, neighbours, rows, length; microseconds by weights and by buckets
@pytest.mark.parametrize("S,entries,l,masks,B,L,weights,buckets", [
    (3000, 1578784, 12, 6571, 50, 200, 24694, 4306),
    (20000, 10549526, 12, 6571, 16, 200, 8754, 3471),
    (3000, 1578784, 12, 6571, 16, 600, 10218, 4354),
    (72000, 38593654, 8, 25, 50, 200, 8010, 4625),
    (20000, 10709526, 8, 25, 50, 200, 2454, 1515),
    (72000, 38881654, 6, 154, 50, 40, 71492, 60154),
    (500, 268118, 11, 4984, 50, 200, 3455, 2096),
    (20000, 10589526, 11, 4984, 50, 40, 3287, 1637),
    (72000, 38161654, 11, 4984, 4, 600, 865, 5010),
    (20000, 10789526, 6, 154, 1, 200, 4939, 11408)])
def test_faster_form(S, entries, l, masks, B, L, weights, buckets):
    model = types.SimpleNamespace(kernel=types.SimpleNamespace(base=types.SimpleNamespace(l=l)))
    index = types.SimpleNamespace(S=S, entries=entries)
    assert explain._row_weights_pay(model, index, B * (L - l + 1), B, masks) == (weights < buckets)
