"""Host codes in pinned memory may be refilled as soon as a call returns: the
copy to the device, queued behind earlier work, is done by then."""

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["predict", "ism", "explain", "variants", "impact"])
@pytest.mark.parametrize("kt", ["gkmrbf", "gkm_esttrunc"])
def test_pinned_codes_are_read_before_the_call_returns(kt, call):
    rng = np.random.default_rng(5)
    m = gk.GkmSVM(syn.random_codes(rng, 3000, 300), rng.normal(size=3000), 0.1, kt,
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    m.use_lmer_table = kt == "gkm_esttrunc"
    x, other = (syn.random_codes(rng, 6, 200) for _ in range(2))
    alt = x.copy()
    alt[:, 100] = (alt[:, 100] + 1) % 4
    run = {"predict": lambda x: m(x), "ism": lambda x: gk.ism(m, x),
           "explain": lambda x: gk.gkmexplain(m, x, mode="hypothetical"),
           "variants": lambda x: m.score_variants(x, alt),
           "impact": lambda x: m.score_variants(x, alt, method="gkmexplain")}[call]
    want = run(x)
    pinned = torch.from_numpy(x).pin_memory()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # ~0.1 s: the copy waits behind it
    got = run(pinned)
    pinned.copy_(torch.from_numpy(other))
    assert torch.equal(got, want)
