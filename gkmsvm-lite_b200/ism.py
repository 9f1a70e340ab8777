"""In silico mutagenesis (ism.py:21-320 of gkmsvm-lite) on the GPU.

Window-delta form: a substitution at p changes only the <= l windows that
cover p.  Kernels with an l-mer table read the changed windows' table weights
and the mutant self-kernels in one fused pass (gkm_ism_table); other kernels
(RBF) count the window pairs each substitution changes once per SV and reduce
over the SVs (gkm_ism_pairs), or where that does not apply or costs more add the
changed windows' index hits to the reference row's kernel values
(gkm_index_mutants).
"""

from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import engine
from ._lib import call, ptr, stream_handle
from .inputs import SeqBatch, device_codes, per_position
from .kernels import RbfKernel, neighbor_count

# Microseconds of an index-path pass of B rows, measured on B200 (l = 8 .. 11, d = 0 ..
# 3, 64 .. 72,000 SVs of 200 .. 350 bp, 1 .. 64 rows of 20 .. 2,000 bp: of 2,697
# shapes pair lists for all are slower than the walk in 1,227, by up to 12 times, by this
# rule in 144, by up to 1.48; 45 are left to the walk that would be faster by up to 1.48).
# Pair lists take the rows one after the other: per row the launches, per SV a block's
# turn, per (SV, position) the mutants' terms, per window pair within dmax + 1 mismatches
# the counters, per list entry the lists.  The walk takes all rows at once: lookups and
# hits of the windows that the mutants change, and the reduction of every (mutant, SV).
_PAIR_ROW_US, _PAIR_SV_US, _PAIR_TERM_US, _PAIR_US, _PAIR_ENTRY_US = 34.0, 6.0e-3, 1.93e-5, 5.7e-6, 1.14e-5
_PAIR_LMER_US = 2.0e-6
_WALK_CALL_US, _WALK_SV_US = 34.5, 6.3e-3
# (unweighted, weighted)
_WALK_POSITION_US, _WALK_TERM_US = (0.116, 0.085), (4.5e-5, 3.9e-5)
_WALK_LOOKUP_US, _WALK_HIT_US = (7.1e-6, 4.8e-6), (1.1e-6, 1.7e-6)


def _pairs_pay(base, index, B: int, L: int, sms: int) -> bool:
    """Whether ISM of B rows of L positions costs less by pair lists (one row
    at a time) than by the walk.  The walk is the faster form for many short
    rows and small neighbourhoods (64 rows of 60 bp, d=1, 72,000 SVs: 18.8
    against 34.4 ms; one of 1,000 bp, d=3: 8.7 against 3.8)."""
    l, S, w = base.l, index.S, int(base.weighted)
    W, n = L - l + 1, 4**l
    near = neighbor_count(l, base.dmax + 1)
    # a block takes an SV at a time, at least one turn each
    blocks = sms * (4 if L <= 512 else 2 if L <= 1024 else 1)
    turns = -(-S // blocks) * blocks
    pairs = W * index.entries / S * turns * near / n
    row = (_PAIR_ROW_US + _PAIR_SV_US * turns + _PAIR_TERM_US * turns * L + _PAIR_US * pairs + _PAIR_ENTRY_US * W * near
           + _PAIR_LMER_US * n)
    changed = 3 * B * L * min(l, W)
    masks = int(index.masks.numel())
    walk = (_WALK_CALL_US + _WALK_SV_US * S + B * L * (_WALK_POSITION_US[w] + _WALK_TERM_US[w] * S)
            + changed * masks * (_WALK_LOOKUP_US[w] * index.tiles + _WALK_HIT_US[w] * index.entries / n))
    return B * row < walk


# Sequences per device pass: ISM outputs [B, 4, L] float64 per pass within this
_BLOCK_BYTES = 1 * 2**30
# Index-path ISM workspace (query rows and K_raw rows of a pass of positions)
_WORKSPACE_BYTES = 3 * 2**29


def ism(model, x, *, lengths=None, batch_size=None, verbose=False) -> torch.Tensor:
    """[B, 4, L] f(mutant) - f(x) for every single-base substitution; 0 past
    each row's length, NaN rows shorter than l (ism.py:21-64)."""
    dev = model._require_gpu()
    batch = SeqBatch.read(x, lengths)
    l = model.kernel.base.l
    short = batch.short(l, "ISM deltas")
    B, L = batch.B, batch.L
    model._plan_lmer_table(5 * l * B * L)
    bs = batch_size if batch_size is not None else max(1, _BLOCK_BYTES // (8 * 4 * L * 3))
    parts = []
    it = range(0, B, bs)
    if verbose:
        from tqdm import tqdm
        it = tqdm(it, desc="ISM")
    for s in it:
        p = batch.part(s, bs)
        parts.append(_ism_rows(model, p.codes, p.lengths, dev))
    out = parts[0] if len(parts) == 1 else torch.cat(parts)
    return per_position(out, batch, short)


def _ism_rows(model, x, lengths, dev, check=True, work=None, table_work=None):
    """[B, 4, L] deltas of one pass (x: host or device codes).  check=False:
    no host synchronisation (the index's exactness check is the caller's)."""
    base = model.kernel.base
    spec = model._spec()
    L = x.shape[-1]
    if L < base.l:
        return torch.full((x.shape[0], 4, L), float("nan"), dtype=torch.float64, device=dev)
    xt = device_codes(x, dev)
    fwd, rc, counts = engine.pack(spec, xt, lengths)
    spec.check_rows(int(fwd.shape[1]))
    table = model._lmer_table_for()
    if table is not None:
        _, raw, diag = engine.table_score(spec, table, fwd, rc, counts, 0.0, base.normalize, want_parts=True)
        return engine.ism_table(spec, table, fwd, counts, L, raw, diag, base.normalize)
    return _ism_index(model, fwd, rc, counts, L, check, work, table_work, engine.known_windows(fwd, lengths, base.l))


def _ism_index(model, fwd, rc, counts, L, check=True, work=None, table_work=None, windows=0):
    kernel = model.kernel
    base = kernel.base
    spec = model._spec()
    index = model._sv_index()
    if index is None:
        raise NotImplementedError("ISM without an l-mer table needs the l-mer index "
                                  "(use_lmer_index=True and a neighbourhood it covers)")
    B, W = fwd.shape
    rbf = isinstance(kernel, RbfKernel)
    gamma = kernel.gamma if rbf else 0.0
    out = torch.empty((B, 4, L), dtype=torch.float64, device=fwd.device)
    pairs = ism_pairs_bytes(model, B, L)
    if work is None:
        work = (torch.empty(pairs, dtype=torch.uint8, device=fwd.device) if pairs
                else ism_workspace(model, B, L, fwd.device))

    def run():
        # the reference rows' K_raw; their scores come from it inside the call
        ref_raw, diag = index.rows(fwd, rc, counts, base.normalize, check=False, work=table_work, windows=windows)
        if base.normalize:
            mut = engine.mutant_diag(spec, fwd, counts, L, diag)
            inv_dx = 1.0 / torch.sqrt(torch.clamp(diag, min=1e-20))
            inv_dmut = 1.0 / torch.sqrt(torch.clamp(mut, min=1e-20))
        else:
            inv_dx = torch.ones(B, dtype=torch.float64, device=fwd.device)
            inv_dmut = torch.ones((4, L, B), dtype=torch.float64, device=fwd.device)
        if 0 < pairs <= work.numel():
            call("gkm_ism_pairs", index.handle, ptr(fwd), ptr(counts), B, W, L, ptr(ref_raw), ptr(inv_dx),
                 ptr(inv_dmut), ptr(model._inv_ds()), ptr(model._sv_coef()), float(gamma), int(rbf), ptr(out),
                 ptr(work), int(work.numel()), stream_handle())
            return out
        call("gkm_index_mutants", index.handle, ptr(fwd), ptr(counts), B, W, L, ptr(ref_raw), None,
             ptr(inv_dx), ptr(inv_dmut), ptr(model._inv_ds()), ptr(model._sv_coef()), float(gamma), int(rbf),
             ptr(out), ptr(work), int(work.numel()), stream_handle())
        return out

    return index.checked(run) if check else run()


def ism_pairs_bytes(model, B: int, L: int) -> int:
    """Workspace bytes of an index-path ISM of B rows x L positions by pair
    lists, 0 where the walk serves it."""
    index = model._sv_index()
    base = model.kernel.base
    n = ctypes.c_int64()
    if _pairs_pay(base, index, B, L, index.sms):
        call("gkm_ism_pairs_workspace", index.handle, L - base.l + 1, L, ctypes.byref(n))
    return n.value


def ism_workspace_bytes(model, B: int, L: int, cap: int = None) -> int:
    """Bytes of an index-path ISM workspace for B rows x L positions: the query
    rows and K_raw rows of as many positions per chunk as fit in cap bytes
    (at least one position's)."""
    lo, hi = ctypes.c_int64(), ctypes.c_int64()
    call("gkm_index_mutants_workspace", model._sv_index().handle, B, L, ctypes.byref(lo), ctypes.byref(hi))
    return max(lo.value, min(hi.value, _WORKSPACE_BYTES if cap is None else cap))


def ism_pass_bytes(model, B: int, positions: int) -> int:
    """Workspace bytes of an index-path ISM pass over `positions` positions of
    B rows (a workspace of this size makes every pass that short)."""
    lo, hi = ctypes.c_int64(), ctypes.c_int64()
    call("gkm_index_mutants_workspace", model._sv_index().handle, B, max(1, int(positions)), ctypes.byref(lo),
         ctypes.byref(hi))
    return hi.value


def ism_workspace(model, B: int, L: int, device, cap: int = None) -> torch.Tensor:
    return torch.empty(ism_workspace_bytes(model, B, L, cap), dtype=torch.uint8, device=device)
