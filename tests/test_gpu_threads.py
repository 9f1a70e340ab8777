"""Two host threads, each on a stream of its own, launching the same kernels with
small and with large dynamic shared memory: neither may lower the limit under the
other's launches, and results are those of the calls made alone."""

import threading

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine

pytestmark = pytest.mark.gpu


def _packed(spec, rows, length, seed):
    x = syn.random_codes(np.random.default_rng(seed), rows, length)
    return engine.pack(spec, torch.from_numpy(x).cuda(), None)


def _count_tables(m, rows, length):
    """1 row takes 20 KB, 32 rows 68 KB."""
    f, _, c = _packed(m._spec(), rows, length, rows)
    index = m._sv_index()
    work = torch.empty(index.table_bytes(*f.shape, 1 << 40), dtype=torch.uint8, device="cuda")

    def call():
        out = torch.empty((rows, index.S), dtype=torch.float64, device="cuda")
        index.table_query(f, c, work=work, raw=out)
        return out

    return call


def _ism(m, rows, length):
    """Pair lists of 60 positions take 7 KB, of 500 positions 54 KB."""
    x = syn.random_codes(np.random.default_rng(length), rows, length)
    return lambda: gk.ism(m, x)


def _self(m, rows, length):
    """The bit planes of 1,000 bases take 0.6 KB, of 120,000 bases 60 KB."""
    spec = m._spec()
    f, r, c = _packed(spec, rows, length, length)
    return lambda: engine.self_kernel(spec, f, r, c)


def _mutants(m, rows, length):
    """The bit planes of 300 bases take 0.5 KB, of 60,000 bases 60 KB."""
    spec = m._spec()
    x = np.zeros((rows, length), np.uint8)
    x[:, :300] = syn.random_codes(np.random.default_rng(length), rows, 300)
    lengths = np.full(rows, 300)
    f, r, c = engine.pack(spec, torch.from_numpy(x).cuda(), lengths)
    d = engine.self_kernel(spec, f, r, c)
    return lambda: engine.mutant_diag(spec, f, c, length, d)


@pytest.mark.parametrize("kind,small,large,n", [
    (_count_tables, (1, 100), (32, 100), 400), (_ism, (1, 60), (1, 500), 40), (_self, (4, 1000), (1, 120_000), 10),
    (_mutants, (1, 300), (1, 60_000), 200)])
def test_two_threads(kind, small, large, n):
    rng = np.random.default_rng(1)
    m = gk.GkmSVM(syn.random_codes(rng, 2000, 300), rng.normal(size=2000), 0.1, "gkmrbf",
                  {"L": 11, "k": 7, "d": 3, "gamma": 1.0}).cuda()
    calls = [kind(m, *small), kind(m, *large)]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    failed, streams = [], [torch.cuda.Stream(), torch.cuda.Stream()]

    def repeat(k):
        try:
            with torch.cuda.stream(streams[k]):
                for _ in range(n):
                    got = calls[k]()
                streams[k].synchronize()
                assert torch.equal(got, want[k])
        except Exception as e:
            failed.append(repr(e))

    ts = [threading.Thread(target=repeat, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed
