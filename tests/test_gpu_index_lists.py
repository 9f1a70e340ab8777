"""Indexes without the count tables' lists: those that only l-mer weights or
kernel columns are read from, and those whose lists do not fit the device."""

import ctypes

import numpy as np
import pytest
import torch

import gkmsvm_lite_b200 as gk
import gkmsvm_lite_b200.synthetic as syn
from gkmsvm_lite_b200 import engine
from gkmsvm_lite_b200._lib import call
from gkmsvm_lite_b200.solver import KernelColumnCache

pytestmark = pytest.mark.gpu

PARAMS = {"L": 11, "k": 7, "d": 3, "gamma": 1.0}


def _pairs_bytes(index, L):
    n = ctypes.c_int64()
    call("gkm_ism_pairs_workspace", index.handle, L - 10, L, ctypes.byref(n))
    return n.value


@pytest.mark.parametrize("kt", ["gkmrbf", "wgkmrbf"])
def test_walk_index(kt):
    rng = np.random.default_rng(8)
    m = gk.GkmSVM(syn.random_codes(rng, 200, 150), rng.normal(size=200), 0.1, kt, PARAMS).cuda()
    full, walk = m._sv_index(), engine.DeviceIndex(m._spec(), *m._sv_packed(), m._masks(), tables=False)
    assert full.table_bytes(4, 90, 1 << 40) > 0 and _pairs_bytes(full, 100) > 0
    assert walk.table_bytes(4, 90, 1 << 40) == 0 and _pairs_bytes(walk, 100) == 0
    assert walk.nbytes < full.nbytes
    f, _, c = engine.pack(m._spec(), torch.from_numpy(syn.random_codes(rng, 4, 100)).cuda(), None)
    assert torch.equal(walk.pairwise(f, c)[0], full.pairwise(f, c)[0])
    walk.close()


@pytest.mark.parametrize("use", ["l-mer table", "explain", "training"])
def test_who_builds_no_lists(use, monkeypatch):
    made = []

    def spy(name, *args):
        made.append(name)
        return call(name, *args)

    monkeypatch.setattr(engine, "call", spy)
    rng = np.random.default_rng(9)
    x = syn.random_codes(rng, 100, 150)
    m = gk.GkmSVM(x, rng.normal(size=100), 0.1, "gkm_esttrunc", PARAMS).cuda()
    if use == "l-mer table":
        m.use_lmer_table = True
        m(x[:3])
    elif use == "explain":
        gk.gkmexplain(m, x[:3])
    else:
        KernelColumnCache(m.kernel, x).compute_columns([0, 1])
    assert "gkm_index_create_walk" in made and "gkm_index_create" not in made


def test_lists_that_do_not_fit():
    """With less and less free memory: wherever the index itself can be built, it
    is built, with its lists or without."""
    rng = np.random.default_rng(10)
    base = gk.CenterWeightedGkmKernel(8, 4, d=3)
    spec = engine.Spec(base, torch.device("cuda"))
    # SVs of one window each: the lists pad them to eight and outweigh the index's own scratch
    x = torch.from_numpy(syn.random_codes(rng, 4_000_000, 8)).cuda()
    fwd, rc, counts = engine.pack(spec, x, None)
    masks = engine.masks_tensor(base, torch.device("cuda"))
    q, _, qc = engine.pack(spec, torch.from_numpy(syn.random_codes(rng, 1, 40)).cuda(), None)
    del x

    def build(tables):
        try:
            return engine.DeviceIndex(spec, fwd, rc, counts, masks, tables=tables)
        except MemoryError:
            return None

    want, with_lists, without = None, 0, 0
    for room in range(640, 140, -20):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        taken = torch.empty(torch.cuda.mem_get_info()[0] - (room << 20), dtype=torch.uint8, device="cuda")
        try:
            walk = build(False)
            if walk is None:
                break
            walk.close()
            index = build(True)
        finally:
            del taken
            torch.cuda.empty_cache()
        assert index is not None, f"{room} MB"
        lists = index.table_bytes(1, 33, 1 << 40) > 0
        with_lists += lists
        without += not lists
        raw = index.pairwise(q, qc)[0]
        want = raw if want is None else want
        assert torch.equal(raw, want)
        index.close()
    assert with_lists and without


@pytest.mark.parametrize("kt,l,d,N,L,tables", [
    ("gkm_esttrunc", 11, 3, 1000, 300, True), ("wgkm", 8, 2, 64, 100, False), ("wgkm", 8, 2, 300, 300, False),
    ("wgkm", 11, 0, 300, 60, False), ("gkm_esttrunc", 11, 3, 100, 400, True), ("wgkm", 11, 3, 64, 1000, True)])
def test_gram_makes_lists_where_they_pay(kt, l, d, N, L, tables, monkeypatch):
    made, lists = [], []

    def spy(name, *args):
        made.append(name)
        return call(name, *args)

    def close(index, real=engine.DeviceIndex.close):
        lists.append(_pairs_bytes(index, 100) > 0)
        real(index)

    monkeypatch.setattr(engine, "call", spy)
    monkeypatch.setattr(engine.DeviceIndex, "close", close)
    x = syn.random_codes(np.random.default_rng(11), N, L)
    kernel = (gk.CenterWeightedGkmKernel if kt == "wgkm" else gk.EstTruncGkmKernel)(l, l - 4, d=d)
    got = gk.compute_gram(kernel, x)
    assert lists == [tables] and ("gkm_count_table_query" in made) == tables
    # the other form
    create = engine.DeviceIndex.__init__
    monkeypatch.setattr(engine.DeviceIndex, "__init__",
                        lambda self, *a, query=None, **kw: create(self, *a, tables=not tables))
    monkeypatch.setattr(engine.DeviceIndex, "tables_pay", lambda *a: not tables)
    monkeypatch.setattr(engine.DeviceIndex, "table_bytes",
                        lambda self, B, W, windows=0, real=engine.DeviceIndex.table_bytes: real(self, B, W, 1 << 40))
    assert np.array_equal(got, gk.compute_gram(kernel, x))


@pytest.mark.parametrize("rows,lists", [(4000, True), (64, None), (0, False)])
def test_lists_for_a_query(rows, lists):
    """An index for a query has lists exactly where one without them says they pay."""
    rng = np.random.default_rng(12)
    m = gk.GkmSVM(syn.random_codes(rng, 200, 150), rng.normal(size=200), 0.1, "wgkmrbf", PARAMS).cuda()
    index = engine.DeviceIndex(m._spec(), *m._sv_packed(), m._masks(), query=(rows, 290, 290 * rows, engine.ROWS_RAW))
    walk = engine.DeviceIndex(m._spec(), *m._sv_packed(), m._masks(), tables=False)
    pays = walk.tables_pay(rows, 290, 290 * rows, engine.ROWS_RAW)
    assert (index.table_bytes(4, 90, 1 << 40) > 0) == pays and lists in (None, pays)
    walk.close()
    f, _, c = engine.pack(m._spec(), torch.from_numpy(syn.random_codes(rng, 4, 100)).cuda(), None)
    want = m._sv_index().pairwise(f, c)[0]
    assert torch.equal(index.pairwise(f, c)[0], want)
    if pays:
        raw = torch.empty((4, 200), dtype=torch.float64, device="cuda")
        work = torch.empty(index.table_bytes(4, 90, 1 << 40), dtype=torch.uint8, device="cuda")
        index.table_query(f, c, work=work, raw=raw)
        assert torch.equal(raw, want)
    index.close()


# SVs, weighted, l, d, rows, length; microseconds of K_raw rows by the walk and by tables
@pytest.mark.parametrize("shape,walk,tables", [
    ((64, 1, 8, 2, 256, 30), 83, 366), ((300, 1, 8, 1, 256, 30), 71, 251), ((3000, 0, 11, 1, 64, 30), 68, 167),
    ((72000, 1, 11, 0, 16, 30), 78, 219), ((64, 0, 11, 3, 1, 100), 800, 59), ((3000, 0, 11, 3, 64, 300), 1619, 279),
    ((300, 0, 8, 2, 64, 100), 544, 117), ((3000, 0, 8, 2, 1, 1000), 694, 55)])
def test_faster_form_of_rows(shape, walk, tables):
    S, weighted, l, d, B, L = shape
    rng = np.random.default_rng(0)
    lengths = rng.integers(200, 351, S)
    m = gk.GkmSVM(syn.ragged_codes(rng, lengths), rng.normal(size=S), 0.1, "wgkmrbf" if weighted else "gkmrbf",
                  {"L": l, "k": l - 4, "d": d, "gamma": 1.0}, sv_lengths=lengths).cuda()
    W = L - l + 1
    assert m._sv_index().tables_pay(B, W, B * W, engine.ROWS_RAW) == (tables < walk)
