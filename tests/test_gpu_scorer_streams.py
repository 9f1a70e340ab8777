"""One scorer or runner called from two streams and from two threads: its
buckets share the count-table workspace, so their passes must not overlap, and a
checked pass is complete when score() returns."""

import threading

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200.batch import BatchedExplain, BatchedIsm, BatchedScorer, DirectScorer
from gkmsvm_lite_b200.engine import DeviceIndex

pytestmark = pytest.mark.gpu


def _model(kt, n_sv):
    rng = np.random.default_rng(1)
    sv = syn.random_codes(rng, n_sv, 300)
    m = gk.GkmSVM(sv, rng.normal(size=n_sv), 0.1, kt, {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    # count tables for every shape (more windows than there are: the walk never looks cheaper)
    index = m._sv_index()
    index.table_bytes = lambda B, W, windows=0: DeviceIndex.table_bytes(index, B, W, 1 << 40)
    index.tables_pay = lambda *a: True
    return m


def _batches(shapes):
    rng = np.random.default_rng(2)
    out = []
    for n, L in shapes:
        ln = rng.integers(L // 2, L + 1, n)
        out.append((syn.ragged_codes(rng, ln), ln))
    return out


def _on_two(run, batches, threads):
    """{batch: results} of run(batch) six times each, every batch on a stream of
    its own: in turn from one thread, or from a thread per batch at once."""
    streams = [torch.cuda.Stream() for _ in batches]
    got = {k: [] for k in range(len(batches))}

    def one(k):
        with torch.cuda.stream(streams[k]):
            got[k].append(run(batches[k]).clone())

    if threads:
        ts = [threading.Thread(target=lambda k=k: [one(k) for _ in range(6)]) for k in range(len(batches))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for _ in range(6):
            for k in range(len(batches)):
                one(k)
    torch.cuda.synchronize()
    return got


@pytest.mark.parametrize("threads", [False, True])
@pytest.mark.parametrize("check", [False, True])
@pytest.mark.parametrize("kt", ["gkmrbf", "wgkmrbf"])
def test_scorer(kt, check, threads):
    m = _model(kt, 6000)
    host = _batches([(1024, 128), (1500, 300)])
    want = [m(x, lengths=ln)[:, 0].cpu().numpy() for x, ln in host]
    batches = [(torch.from_numpy(x).cuda(), torch.from_numpy(ln).cuda()) for x, ln in host]
    s = BatchedScorer(m)
    got = _on_two(lambda b: s.score(*b, check=check), batches, threads)
    assert all(g.work is not None for g in s._graphs.values()) and len(s._graphs) == 2
    for k, w in enumerate(want):
        assert len(got[k]) == 6
        for g in got[k]:
            # (another order of the sum over the SVs)
            np.testing.assert_allclose(g.cpu().numpy(), w, rtol=1e-11, atol=1e-11)


@pytest.mark.parametrize("threads", [False, True])
@pytest.mark.parametrize("kind", ["ism", "explain"])
def test_runner(kind, threads):
    m = _model("gkmrbf", 3000)
    host = _batches([(8, 64), (8, 200)])
    if kind == "ism":
        runner, call = BatchedIsm(m), lambda x, ln: gk.ism(m, x, lengths=ln)
    else:
        runner, call = BatchedExplain(m), lambda x, ln: gk.gkmexplain(m, x, lengths=ln, mode="hypothetical")
    want = [call(x, ln).cpu().numpy() for x, ln in host]
    batches = [(torch.from_numpy(x).cuda(), torch.from_numpy(ln).cuda()) for x, ln in host]
    got = _on_two(lambda b: runner(*b), batches, threads)
    for k, w in enumerate(want):
        assert len(got[k]) == 6
        for g in got[k]:
            np.testing.assert_allclose(g.cpu().numpy(), w, rtol=1e-9, atol=1e-12 * max(1.0, np.abs(w).max()))


@pytest.mark.parametrize("scorer", [BatchedScorer, DirectScorer])
def test_a_checked_pass_is_complete(scorer):
    m = _model("gkmrbf", 3000)
    s = scorer(m)
    x = torch.from_numpy(syn.random_codes(np.random.default_rng(3), 64, 200)).cuda()
    s.score(x)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        s.score(x)
    assert stream.query()
