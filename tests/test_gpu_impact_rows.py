"""GkmExplain impacts through the index walk normalise by the reference alleles
and compute no other self-kernels."""

import numpy as np
import pytest

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", ["gkmrbf", "wgkmrbf"])
@pytest.mark.parametrize("n", [1, 7])
def test_self_kernels_of_the_references_only(kt, n, monkeypatch):
    rng = np.random.default_rng(n)
    m = gk.GkmSVM(syn.random_codes(rng, 100, 150), rng.normal(size=100), 0.1, kt,
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    ref = syn.random_codes(rng, n, 90)
    alt = ref.copy()
    alt[:, 40] = (alt[:, 40] + 1) % 4
    tables = m.score_variants(ref, alt, method="gkmexplain").cpu().numpy()
    rows, real = [], engine.self_kernel
    monkeypatch.setattr(engine, "self_kernel", lambda spec, f, *a, **k: rows.append(f.shape[0]) or real(spec, f, *a, **k))
    monkeypatch.setattr(engine.DeviceIndex, "table_bytes", lambda *a: 0)  # the walk
    walk = m.score_variants(ref, alt, method="gkmexplain").cpu().numpy()
    assert rows == [n]
    np.testing.assert_allclose(walk, tables, rtol=1e-12, atol=1e-13)
