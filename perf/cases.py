"""Timed cases of the framework: scoring, variant effects, in silico mutagenesis,
GkmExplain attributions and Gram matrices through the public entry points.

Sequences are i.i.d. bases at GC 0.42 (the repository's synthetic workloads);
models have 2,000 to 72,000 support vectors of 200..500 bp, queries are
50..2,000 bp.  The values of each case:

  entry    what is called: "predict" model(x) on host codes, "batched"
           BatchedScorer.score on device codes, "impact" / "variants"
           score_variants with method "gkmexplain" / "kernel", "ism",
           "explain" (hypothetical GkmExplain), "gram" compute_gram
  kernel   kernel type (LS-GKM -t name), l, k, d and gamma its parameters
  n_sv     support vectors (gram: none)
  rows     query sequences (variants: pairs), lengths log-uniform lo..hi, the
           first row hi long
  table    True: a linear model scores through its l-mer table
"""

import math

import numpy as np
import torch

import gkmsvm_lite_b200 as gk
from gkmsvm_lite_b200.batch import BatchedScorer

RBF = ("gkmrbf", "wgkmrbf", "gkm_cnt_rbf")
WEIGHTED = ("wgkm", "wgkmrbf")


def _case(name, entry, kernel, rows, lo, hi, n_sv=72000, l=11, k=7, gamma=2.0, table=False):
    c = {"entry": entry, "kernel": kernel, "l": l, "k": k, "d": 3, "gamma": gamma, "n_sv": n_sv, "rows": rows,
         "lo": lo, "hi": hi, "table": table}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one sequence scored on its own: an interactive call, a lone request of a server
        _case("predict-one", "predict", "gkmrbf", 1, 300, 300),
        # a chromatin-accessibility peak set against a large trained model, host arrays in
        _case("predict-1000", "predict", "gkmrbf", 1000, 300, 300, gamma=1.0),
        # the batched form of a scan over sequences of every length
        _case("batched-ragged", "batched", "gkmrbf", 2048, 50, 2000),
        # the same with centre-weighted windows (-t 5), the served model
        _case("batched-weighted", "batched", "wgkmrbf", 512, 50, 2000, gamma=1.0),
        # a small model with an even window length (-t 6)
        _case("predict-small-model", "predict", "gkm_cnt_rbf", 1000, 290, 300, n_sv=2000, l=10, k=6, gamma=1.0),
        # LS-GKM's default kernel through the l-mer table, the bulk scoring of a linear model
        _case("batched-table", "batched", "gkm_esttrunc", 8192, 50, 2000, table=True),
        # every substitution of a peak set, linear model
        _case("ism-linear", "ism", "gkm_esttrunc", 128, 300, 300, table=True),
        # every substitution of one sequence, RBF model
        _case("ism-rbf", "ism", "wgkmrbf", 1, 500, 500, gamma=1.0),
        # attributions of a peak set, linear model
        _case("explain-linear", "explain", "gkm_esttrunc", 512, 1000, 1000),
        # attributions of a few sequences, RBF model
        _case("explain-rbf", "explain", "gkmrbf", 4, 300, 600, gamma=1.0),
        # GkmExplain impact of variants (SNVs and indels), RBF model
        _case("impact-rbf", "impact", "gkmrbf", 96, 300, 300, gamma=1.0),
        # the Gram matrix a training run needs, host to host
        _case("gram-weighted", "gram", "wgkm", 2000, 100, 1000, n_sv=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["predict", "predict", "batched", "batched", "variants", "impact", "ism", "ism", "explain",
                        "explain", "gram"])
    if entry == "gram":
        return _case(None, entry, rng.choice(["wgkm", "gkm_esttrunc", "gkmrbf"]), _log_int(rng, 100, 2000), 100,
                     _log_int(rng, 300, 1000), n_sv=0, gamma=1.0)
    kernel = rng.choice(["gkm_esttrunc", "gkmrbf", "wgkm", "wgkmrbf"])
    n_sv = _log_int(rng, 2000, 72000)
    hi = _log_int(rng, 60, 2000)
    lo = rng.choice([hi, max(50, hi // 4)])
    l, k = rng.choice([(11, 7), (11, 7), (10, 6)])
    most = {"predict": 1000, "batched": 2048, "variants": 100, "impact": 64, "ism": 64, "explain": 128}[entry]
    rbf = kernel in RBF
    if rbf and entry == "ism":
        most, hi, lo = 2, min(hi, 500), min(lo, 500)
    if rbf and entry == "explain":
        most = 4
    if kernel == "wgkmrbf":
        most = min(most, 256)
    return _case(None, entry, kernel, _log_int(rng, 1, most), lo, hi, n_sv=n_sv, l=l, k=k, gamma=rng.choice([1.0, 2.0]),
                 table=entry in ("batched", "ism") and not rbf)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _codes(g, lengths):
    """[n, max] uint8 base codes at GC 0.42, 0 past each row's length."""
    u = torch.rand((len(lengths), int(lengths.max())), generator=g, device="cuda")
    c = ((u > 0.29).to(torch.uint8) + (u > 0.5).to(torch.uint8) + (u > 0.71).to(torch.uint8))
    past = torch.arange(u.shape[1], device="cuda")[None, :] >= torch.from_numpy(lengths).cuda()[:, None]
    return c.masked_fill_(past, 0).cpu().numpy()


def _log_uniform(rng, n, lo, hi):
    return np.clip(np.floor(np.exp(rng.uniform(math.log(lo), math.log(hi + 1), n))), lo, hi).astype(np.int64)


def _variants(rng, x, xl):
    """Alternative alleles: an SNV (80 %) or an indel of 1..10 bp per row."""
    alt = np.zeros((x.shape[0], x.shape[1] + 10), np.uint8)
    al = np.empty(len(xl), np.int64)
    for i, n in enumerate(xl):
        s, p, size = x[i, :n], int(rng.integers(1, n - 1)), int(rng.integers(1, 11))
        kind = rng.random()
        if kind < 0.8 or n < 40:
            s = s.copy()
            s[p] = (s[p] + 1 + int(rng.integers(0, 3))) % 4
        elif kind < 0.9:
            s = np.concatenate([s[:p], rng.integers(0, 4, size).astype(np.uint8), s[p:]])
        else:
            s = np.concatenate([s[:p], s[p + size:]])
        alt[i, :len(s)] = s
        al[i] = len(s)
    return alt, al


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    i = {}
    if case["n_sv"]:
        i["svl"] = rng.integers(200, 501, case["n_sv"]).astype(np.int64)
        i["sv"] = _codes(g, i["svl"])
        i["coef"] = rng.normal(0.0, 0.1, case["n_sv"])
    i["xl"] = _log_uniform(rng, case["rows"], case["lo"], case["hi"])
    i["xl"][0] = case["hi"]
    i["x"] = _codes(g, i["xl"])
    if case["entry"] in ("variants", "impact"):
        i["alt"], i["al"] = _variants(rng, i["x"], i["xl"])
    return i


def _params(case):
    return {"L": case["l"], "k": case["k"], "d": case["d"], "gamma": case["gamma"]}


def prepare(case, seed):
    i = _inputs(case, seed)
    s = {"case": case, **i}
    if case["entry"] == "gram":
        s["kernel"] = {"wgkm": gk.CenterWeightedGkmKernel, "gkm_esttrunc": gk.EstTruncGkmKernel,
                       "gkmrbf": gk.RbfGkmKernel}[case["kernel"]](case["l"], case["k"], d=case["d"])
        return s
    m = gk.GkmSVM(i["sv"], i["coef"], 0.1, case["kernel"], _params(case), sv_lengths=i["svl"]).cuda()
    if case["table"]:
        m.use_lmer_table = True
    s["model"] = m
    m(np.zeros((1, 64), np.uint8))  # a trained model in service: its device state is built
    if case["entry"] == "batched":
        s["scorer"] = BatchedScorer(m)
        s["xd"] = torch.from_numpy(i["x"]).cuda()
        s["ld"] = torch.from_numpy(i["xl"]).cuda()
        for _ in range(2):  # a scorer in service has captured this batch shape
            s["scorer"].score(s["xd"], torch.full_like(s["ld"], case["l"]))
    return s


def run(s):
    case = s["case"]
    entry = case["entry"]
    if entry == "predict":
        return s["model"](s["x"], lengths=s["xl"])
    if entry == "batched":
        return s["scorer"].score(s["xd"], s["ld"])
    if entry in ("variants", "impact"):
        return s["model"].score_variants(s["x"], s["alt"], ref_lengths=s["xl"], alt_lengths=s["al"],
                                         method="kernel" if entry == "variants" else "gkmexplain")
    if entry == "ism":
        return gk.ism(s["model"], s["x"], lengths=s["xl"])
    if entry == "explain":
        return gk.gkmexplain(s["model"], s["x"], lengths=s["xl"], mode="hypothetical", batch_size=case["rows"])
    return gk.compute_gram(s["kernel"], s["x"], lengths=s["xl"])


def work(case):
    mean = (case["lo"] + case["hi"]) / 2 if case["hi"] < 2 * case["lo"] else \
        (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    rows, n_sv = case["rows"], case["n_sv"]
    entry = case["entry"]
    if entry == "gram":
        return {"bytes": rows * mean + 8 * rows * rows, "flops": 2 * 4 * rows * rows / 2}
    alleles = 2 if entry in ("variants", "impact") else 1
    bytes_ = alleles * rows * mean + 8 * rows
    linear = case["kernel"] not in RBF
    sv_bytes = 350 * n_sv
    if entry in ("ism", "explain"):
        bytes_ += 8 * 4 * rows * mean
    if linear:  # sum over windows of one weight per l-mer
        sv_bytes = min(sv_bytes, 8 * rows * mean)
        flops = 2 * alleles * rows * mean * (4 * case["l"] if entry in ("ism", "explain") else 1)
    else:  # every (sequence, support vector) value: 4 levels weighted, normalised, summed
        mutants = 3 * mean if entry == "ism" else 1
        flops = 12.0 * alleles * rows * mutants * n_sv
    return {"bytes": bytes_ + sv_bytes, "flops": flops}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits, plain torch
# ---------------------------------------------------------------------------


def _pair_weights(case):
    """h(m), m = 0..l, zero past d."""
    l, k, d = case["l"], case["k"], case["d"]
    if case["kernel"] == "gkm_cnt_rbf":
        return [float(math.comb(l - m, k)) if m <= d else 0.0 for m in range(l + 1)]
    old, new = [[1.0] * (k + 1) for _ in range(k + 1)], [[1.0] * (k + 1) for _ in range(k + 1)]
    for il in range(1, l + 1):
        for ik in range(1, k + 1):
            new[ik][0] = old[ik][0] + 3 * old[ik - 1][0]
            for jm in range(1, ik + 1):
                new[ik][jm] = new[ik - 1][jm - 1] * (ik - il) / ik
        old, new = new, old
    wm = [old[k][i] / (math.comb(l, k) * 4**l) for i in range(k + 1)]
    est = np.array([sum(wm[i] * math.comb(l - m, k - i) * math.comb(m, i)
                        for i in range(min(m, k) + 1) if l - m >= k - i) for m in range(l + 1)])
    low = np.flatnonzero(est < 1e-50)
    if len(low):
        est[low[0]:] = 0.0
    h = []
    for m in range(l + 1):
        # l-mers by their distances (a, b) to two l-mers m apart: one factor per position
        n = np.zeros((l + 1, l + 1))
        n[0, 0] = 1.0
        for pos in range(l):
            t = np.zeros_like(n)
            if pos < l - m:
                t += n
                t[1:, 1:] += 3 * n[:-1, :-1]
            else:
                t[1:] += n[:-1]
                t[:, 1:] += n[:, :-1]
                t[1:, 1:] += 2 * n[:-1, :-1]
            n = t
        h.append(float(est @ n @ est) if m <= d else 0.0)
    return h


def _windows(x, xl, l):
    """[n, W] l-mer ids (base j at digit j) of rows of codes, and [n, W] bool: a window of the row."""
    x = torch.as_tensor(x).cuda().long()
    W = x.shape[1] - l + 1
    u = sum(x[:, j:j + W] << (2 * j) for j in range(l))
    ok = torch.arange(W, device="cuda")[None, :] < (torch.as_tensor(xl).cuda() - l + 1)[:, None]
    return u, ok


def _rc(u, l):
    r = torch.zeros_like(u)
    for j in range(l):
        r |= (3 - ((u >> (2 * j)) & 3)) << (2 * (l - 1 - j))
    return r


def _weights(case, ok):
    """[n, W] float64 window weights (0: no window)."""
    if case["kernel"] not in WEIGHTED:
        return ok.double()
    n = ok.sum(dim=1, keepdim=True)
    dist = (n // 2 - torch.arange(ok.shape[1], device="cuda")[None, :]).abs().double()
    return torch.floor(50 * torch.exp(-math.log(2.0) * dist / 50.0) + 1).clamp(max=50.0) * ok


def _spread(vec, l, levels):
    """[4^l]: sum over l-mers v of levels[m(u, v)] vec[v], digit by digit."""
    d = len(levels) - 1
    p = [vec] + [torch.zeros_like(vec) for _ in range(d)]
    for j in range(l):
        p = [t.view(-1, 4, 4**j) for t in p]
        other = [t.sum(dim=1, keepdim=True) - t for t in p[:-1]]
        p = [(p[m] + other[m - 1] if m else p[0]).reshape(-1) for m in range(d + 1)]
    return sum(float(c) * t for c, t in zip(levels, p))


def _self(case, x, xl):
    """[n] K(x, x): every pair of windows, forward and reverse complement."""
    l = case["l"]
    h = torch.tensor(_pair_weights(case)[::-1], dtype=torch.float64, device="cuda")  # by matches
    xl = np.asarray(xl)
    out = torch.zeros(len(xl), dtype=torch.float64, device="cuda")
    order = np.argsort(-xl, kind="stable")
    s = 0
    while s < len(order):
        width = int(xl[order[s]])
        n = max(1, int(2**25 // width**2))
        rows = order[s:s + n]
        s += n
        u, ok = _windows(np.asarray(x)[rows][:, :width], xl[rows], l)
        w = _weights(case, ok)
        digits = torch.arange(l, device="cuda") * 2

        def onehot(v):
            return torch.nn.functional.one_hot((v[..., None] >> digits) & 3, 4).float().flatten(2)

        f = onehot(u)
        for other in (f, onehot(_rc(u, l))):
            k = h[torch.bmm(f, other.transpose(1, 2)).round_().long()]
            out[torch.as_tensor(rows).cuda()] += torch.bmm(torch.bmm(w[:, None], k), w[:, :, None])[:, 0, 0]
    return out


class _Exact:
    """K_raw rows of query sequences against a column set."""

    def __init__(self, case, y, yl):
        self.case, self.l = case, case["l"]
        self.h = _pair_weights(case)[:case["d"] + 1]
        u, ok = _windows(y, yl, self.l)
        self.w = _weights(case, ok)
        self.u = torch.where(ok, u, torch.zeros_like(u))
        self.rc = _rc(torch.arange(4**self.l, device="cuda"), self.l)
        self.diag = _self(case, y, yl)

    def weights(self, c):
        """[4^l] sum of c[s] over the windows of column s and their reverse complements."""
        v = torch.zeros(4**self.l, dtype=torch.float64, device="cuda")
        v.index_add_(0, self.u.reshape(-1), (self.w * c[:, None]).reshape(-1))
        return v + v[self.rc]

    def raw(self, x, xl):
        u, ok = _windows(np.asarray(x)[None, :], [int(xl)], self.l)
        v = torch.zeros(4**self.l, dtype=torch.float64, device="cuda")
        v.index_add_(0, u[0], _weights(self.case, ok)[0])
        t = _spread(v, self.l, self.h)
        t = t + t[self.rc]
        return (t[self.u] * self.w).sum(dim=1)


def _scores(case, i, x, xl):
    """[n] decision values without the bias."""
    e = _Exact(case, i["sv"], i["svl"])
    coef = torch.from_numpy(i["coef"]).cuda()
    dx = _self(case, x, xl)
    if case["kernel"] in RBF:
        z = 1.0 / torch.sqrt(e.diag)
        return torch.stack([(coef * torch.exp(case["gamma"] * (e.raw(r, n) * z / torch.sqrt(q) - 1.0))).sum()
                            for r, n, q in zip(x, xl, dx)])
    t = _spread(e.weights(coef / torch.sqrt(e.diag)), e.l, e.h)
    u, ok = _windows(x, xl, e.l)
    return (t[u] * _weights(case, ok)).sum(dim=1) / torch.sqrt(dx)


def _explain(case, i):
    l, d = case["l"], case["d"]
    h = _pair_weights(case)
    e = _Exact(case, i["sv"], i["svl"])
    c = torch.from_numpy(i["coef"]).cuda() / torch.sqrt(e.diag)
    dx = _self(case, i["x"], i["xl"])
    u, ok = _windows(i["x"], i["xl"], l)
    wx = _weights(case, ok)
    B, W = u.shape
    same = [h[m] / (l - m) for m in range(d + 1)]
    diff = [0.0] + [h[m - 1] / (l - m + 1) for m in range(1, d + 1)]
    masks = [((), 0)]
    for j in range(l):
        masks += [(p + ((j, a),), x | a << (2 * j)) for p, x in masks if len(p) < d for a in (1, 2, 3)]
    out = torch.zeros((B, 4, W + l - 1), dtype=torch.float64, device="cuda")
    groups = [(b, b + 1) for b in range(B)] if case["kernel"] in RBF else [(0, B)]
    for b0, b1 in groups:
        cw = c
        if case["kernel"] in RBF:
            k = e.raw(i["x"][b0], i["xl"][b0]) / torch.sqrt(e.diag * dx[b0])
            g = case["gamma"]
            cw = c * torch.where(k > 0, (torch.exp(g * (k - 1)) - math.exp(-g)) / k.clamp(min=1e-300), 0.0)
        v = e.weights(cw)
        ub = u[b0:b1].reshape(-1)
        acc = torch.zeros((l, 4, ub.numel()), dtype=torch.float64, device="cuda")  # by position, mask digit
        for pos, x in masks:
            val = v[ub ^ x]
            acc[:, 0] += same[len(pos)] * val
            for j, a in pos:
                acc[j, 0] -= same[len(pos)] * val
                acc[j, a] += diff[len(pos)] * val
        acc = (acc * wx[b0:b1].reshape(-1)).view(l, 4, b1 - b0, W)
        for j in range(l):
            base = (u[b0:b1] >> (2 * j)) & 3
            for a in range(4):
                out[b0:b1, :, j:j + W].scatter_add_(1, (base ^ a)[:, None], acc[j, a][:, None])
    return out / torch.sqrt(dx)[:, None, None]


def exact(case, seed):
    i = _inputs(case, seed)
    entry = case["entry"]
    x, xl = i["x"], i["xl"]
    rbf = case["kernel"] in RBF
    if entry in ("predict", "batched"):
        out = _scores(case, i, x, xl) + 0.1
        return out[:, None] if entry == "predict" else out
    if entry == "variants":
        r = np.pad(x, ((0, 0), (0, i["alt"].shape[1] - x.shape[1])))
        return (_scores(case, i, i["alt"], i["al"]) - _scores(case, i, r, xl))[:, None]
    if entry == "ism":
        if float((xl**3).sum()) > 1.2e10:
            return None
        B, L = x.shape
        m = np.repeat(x, 4 * L, axis=0)
        n = np.arange(B * 4 * L)
        m[n, n % L] = (n // L) % 4
        ml = np.repeat(xl, 4 * L)
        live = n % L < ml
        out = torch.zeros(B * 4 * L, dtype=torch.float64, device="cuda")
        changed = np.flatnonzero(live & (m[n, n % L] != np.repeat(x, 4 * L, axis=0)[n, n % L]))
        both = _scores(case, i, np.concatenate([m[changed], x]), np.concatenate([ml[changed], xl]))
        ref = both[len(changed):][torch.from_numpy(changed // (4 * L)).cuda()]
        out[torch.from_numpy(changed).cuda()] = both[:len(changed)] - ref
        return out.view(B, 4, L)
    if entry == "explain":
        return _explain(case, i)
    if entry == "impact":
        e = _Exact(case, i["sv"], i["svl"])
        coef = torch.from_numpy(i["coef"]).cuda()
        out = []
        for r, n, a, na, q in zip(x, xl, i["alt"], i["al"], _self(case, x, xl)):
            k = e.raw(r, n)
            z = torch.sqrt(e.diag * q)
            dk, k = (e.raw(a, na) - k) / z, k / z
            if rbf:
                g = case["gamma"]
                dk = dk * torch.where(k > 0, (torch.exp(g * (k - 1)) - math.exp(-g)) / k.clamp(min=1e-300), 0.0)
            out.append((coef * dk).sum())
        return torch.stack(out)[:, None]
    e = _Exact(case, x, xl)
    k = torch.stack([e.raw(r, n) for r, n in zip(x, xl)]) / torch.sqrt(e.diag[:, None] * e.diag[None, :])
    k = torch.exp(k - 1.0) if rbf else k
    return k.cpu().numpy()
