"""The work this engine is run for, as cases that can be timed and checked.

Every case is one call sequence of the public Python binding on seeded
synthetic cohorts: dosages x = clip(Binomial(2, maf) + U(-0.05, 0.05), 0, 2)
rounded to 0.001 (or three genotype probabilities per SNP), covariates
[intercept, sex, age, PCs...], traits with one causal SNP each and missing
phenotypes in patterns.  Matrices are variable-major (v, n) float32, the
layout of .fvd files.

Kinds of case:

* ``scan``: an engine that holds its covariates (and its trait block unless
  ``new_traits``) scans one SNP block, in device memory or in pinned host
  memory, and gives the stored rows;
* ``serve``: a server with a resident genotype matrix serves a few requests,
  each with its own individuals, covariates, traits and SNP range;
* ``noalloc``: the entry point for callers that cannot allocate GPU memory.

Rows are stored at the genome-wide threshold (P < 5e-8: |t| > 5.4513), as a
scan of thousands of traits is in practice, or every test is stored (``-f``).
The causal effects are 0.5 standard deviations and more in small cohorts, well
clear of the threshold.
The number of stored rows depends on the data, so a case gives its rows in a
table of fixed size (unused entries zero) with their count beside it.
The file front end (``oa_solve``) is not among the cases: it writes its
numbers as rounded text.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from omicabelnomm_b200 import engine as E
from omicabelnomm_b200 import serve as S

T_GENOME_WIDE = 5.4513
T_NOMINAL = 1.6449
MIN_R2 = 1e-6

_SCAN = {"kind": "scan", "precision": "mixed", "n": 10000, "l": 4, "r": 1, "t": 1000, "m": 20000, "patterns": 20,
         "miss": 0.10, "zipf": False, "nan_snps": 0.0, "collinear": False, "model": "dosage", "source": "device",
         "store": "genome", "cov": False, "new_traits": False}


def _scan(**over):
    return {**_SCAN, **over}


def listed():
    return [
        # one trait, one SNP block of the reference's size (500): the smallest call a user's loop makes
        _scan(name="one-trait-block", precision="plain", n=1000, l=3, t=1, m=500, patterns=1),
        # the reference's own scale (n = 1,000, 100 traits, 5 % of each trait missing at random: every trait
        # is a pattern of its own), default precision
        _scan(name="plain-own-patterns", precision="plain", n=1000, l=3, t=100, m=10000, patterns=0, miss=0.05),
        # the default precision at omics scale, a block of an .fvd file with a ragged last chunk
        _scan(name="plain-omics", precision="plain", m=60000),
        # a cohort whose size is no multiple of anything, typed SNPs with missing calls, a new trait block
        # for every pass (the trait-block loop of a scan)
        _scan(name="plain-odd-cohort", precision="plain", n=4713, l=6, t=333, m=7777, patterns=11, nan_snps=0.03,
              new_traits=True),
        # every test and every covariate term stored (-f -i), additive model from genotype probabilities
        _scan(name="plain-all-terms", precision="plain", n=2003, l=4, t=64, m=1500, patterns=6, model="probs",
              store="all", cov=True),
        # omics scale, tensor-core precision: the scan this framework is for
        _scan(name="mixed-omics", m=500000),
        # an odd cohort with a near-collinear covariate
        _scan(name="mixed-odd-cohort", n=9973, l=5, t=1000, m=60000, collinear=True),
        # a handful of traits over many SNPs (a plain GWAS): reading the genotypes is all there is
        _scan(name="mixed-few-traits", n=12347, l=6, t=7, m=100000, patterns=3),
        # SNP x sex interactions and 150 uneven missingness patterns
        _scan(name="mixed-interactions", n=8000, l=5, r=2, t=2000, m=20000, patterns=150, miss=0.15, zipf=True),
        # genotypes arriving from host memory, as a reader of files larger than HBM feeds them
        _scan(name="mixed-host-blocks", m=20000, source="host"),
        # four requests at once against a resident genotype matrix
        {"name": "serve-requests", "kind": "serve", "n_total": 20000, "m_total": 60000, "requests": 4, "mix": 11,
         "n_lo": 2000, "t_hi": 500},
        # a plug-in that cannot allocate device memory
        {"name": "plug-in-block", "kind": "noalloc", "n": 2000, "l": 4, "r": 1, "t": 200, "m": 4000, "miss": 0.05},
    ]


# n * r * m * t of the largest drawn scans in each precision (below the largest listed ones)
_COST = {"plain": 1.5e11, "mixed": 1.5e12}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan"] * 8 + ["serve", "noalloc"])
    if kind == "serve":
        return {"kind": "serve", "n_total": rng.randint(8000, 20000), "m_total": _log(rng, 15000, 60000),
                "requests": rng.randint(1, 5), "mix": rng.randint(0, 10 ** 6), "n_lo": 2000, "t_hi": 500}
    if kind == "noalloc":
        n = _log(rng, 400, 4000)
        t = _log(rng, 2, 300)
        return {"kind": "noalloc", "n": n, "l": rng.randint(2, 8), "r": 1,
                "t": t, "m": max(16, min(_log(rng, 100, 6000), 4_000_000 // t - 1)), "miss": rng.choice([0.0, 0.03, 0.08])}
    precision = rng.choice(["plain", "mixed"])
    n = _log(rng, 500, 15000)
    r = rng.choice([1, 1, 1, 1, 1, 2, 2])
    t = _log(rng, 1, 2000)
    cap = _COST[precision] / (n * r * t)
    m = max(300, int(min(_log(rng, 500, 200000), cap, 2.0e9 / (n * r))))
    store = "all" if m * t <= 150000 and rng.random() < 0.5 else "genome"
    patterns = rng.choice([1, 3, 8, 20, 40]) if t > 3 else 1
    if t <= 128 and rng.random() < 0.25:
        patterns = 0
    model = "dosage"
    if m * n * 3 <= 1.0e9 and r == 1 and rng.random() < 0.2:
        model = "probs"
    elif r == 2 and rng.random() < 0.4:
        model = "inter"
    return _scan(precision=precision, n=n, l=rng.randint(2, 8), r=r, t=t, m=m, patterns=min(patterns, t),
                 miss=rng.choice([0.02, 0.05, 0.10, 0.15]), nan_snps=rng.choice([0.0, 0.0, 0.02]), model=model,
                 source="host" if m * n * r <= 3.0e8 and rng.random() < 0.2 else "device", store=store,
                 cov=store == "all" and rng.random() < 0.5, new_traits=rng.random() < 0.2)


# ---------------------------------------------------------------------------
# inputs (from the seed alone)
# ---------------------------------------------------------------------------
def _gen(seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    return g


def _covariates(g, n, l, dev, collinear=False):
    cols = [torch.ones(n, device=dev), (torch.rand(n, generator=g, device=dev) < 0.5).float()]
    while len(cols) < l:
        z = torch.randn(n, generator=g, device=dev)
        cols.append(50.0 + 10.0 * z if len(cols) == 2 else z)
    if collinear and l >= 4:
        cols[l - 1] = cols[2] + 1e-3 * torch.randn(n, generator=g, device=dev)
    return torch.stack(cols[:l]).contiguous()


def _dosages(g, n, m, dev, nan_snps=0.0):
    X = torch.empty((m, n), dtype=torch.float32, device=dev)
    for c0 in range(0, m, 8192):
        c1 = min(m, c0 + 8192)
        maf = 0.01 + 0.49 * torch.rand((c1 - c0, 1), generator=g, device=dev)
        x = (torch.rand((c1 - c0, n), generator=g, device=dev) < maf).float()
        x += (torch.rand((c1 - c0, n), generator=g, device=dev) < maf).float()
        x += 0.1 * torch.rand((c1 - c0, n), generator=g, device=dev) - 0.05
        torch.div(torch.round(x.clamp_(0.0, 2.0).mul_(1000.0)), 1000.0, out=X[c0:c1])
        if nan_snps > 0:   # a share of the SNPs is typed with 1 % of the calls missing
            typed = torch.rand((c1 - c0, 1), generator=g, device=dev) < nan_snps
            miss = torch.rand((c1 - c0, n), generator=g, device=dev) < 0.01
            X[c0:c1][typed & miss] = float("nan")
    return X


def _probabilities(g, n, m, dev):
    """(3 m, n): P(AA), P(AB), P(BB) of each SNP, rounded to 0.001."""
    P = torch.empty((m, 3, n), dtype=torch.float32, device=dev)
    for c0 in range(0, m, 2048):
        c1 = min(m, c0 + 2048)
        maf = 0.02 + 0.48 * torch.rand((c1 - c0, 1), generator=g, device=dev)
        cls = (torch.rand((c1 - c0, n), generator=g, device=dev) < maf).long()
        cls += (torch.rand((c1 - c0, n), generator=g, device=dev) < maf).long()
        e = 0.3 * torch.rand((c1 - c0, n), generator=g, device=dev)
        s = torch.rand((c1 - c0, n), generator=g, device=dev)
        # the class of the genotype gets 1 - e; of the other two, the one listed first gets s of e
        P[c0:c1, 0] = torch.where(cls == 2, 1.0 - e, e * s)
        P[c0:c1, 1] = torch.where(cls == 1, 1.0 - e, e * torch.where(cls == 2, s, 1.0 - s))
        P[c0:c1, 2] = torch.where(cls == 0, 1.0 - e, e * (1.0 - s))
    torch.div(torch.round(P * 1000.0), 1000.0, out=P)
    return P.view(3 * m, n)


def _pattern_of_traits(g, t, patterns, zipf, dev):
    if not zipf:
        return torch.arange(t, device=dev) % patterns
    w = torch.arange(1, patterns + 1, dtype=torch.float64) ** -1.2
    size = torch.clamp((w / w.sum() * t).floor().long(), min=1)
    size[0] += t - int(size.sum())
    pat = torch.repeat_interleave(torch.arange(patterns), size).to(dev)
    return pat[torch.randperm(t, generator=g, device=dev)]


def _traits(g, XL, causal, t, patterns, miss, zipf, dev):
    """Traits XL b + effect * (standardised x_causal) + noise with missing phenotypes; patterns = 0: every
    trait its own."""
    n = XL.shape[1]
    causal = causal - torch.nanmean(causal, dim=1, keepdim=True)
    causal = torch.nan_to_num(causal) / torch.sqrt(torch.nanmean(causal * causal, dim=1, keepdim=True))
    b = torch.randn((t, XL.shape[0]), generator=g, device=dev)
    sd = torch.sqrt(0.5 + 1.5 * torch.rand((t, 1), generator=g, device=dev))
    Y = b @ XL + max(0.5, 17.0 / math.sqrt(n)) * causal + sd * torch.randn((t, n), generator=g, device=dev)
    if patterns == 0:
        Y[torch.rand((t, n), generator=g, device=dev) < miss] = float("nan")
    else:
        frac = miss * torch.rand((patterns, 1), generator=g, device=dev)
        gone = torch.rand((patterns, n), generator=g, device=dev) < frac
        Y[gone[_pattern_of_traits(g, t, patterns, zipf, dev)]] = float("nan")
    return Y.contiguous()


def _scan_inputs(c, seed):
    dev = torch.device("cuda")
    g = _gen(seed, dev)
    n, m, t, r = c["n"], c["m"], c["t"], c["r"]
    XL = _covariates(g, n, c["l"], dev, c["collinear"])
    inter = XL[1:r].contiguous() if c["model"] == "inter" else None   # SNP x sex
    if c["model"] == "probs":
        XR = _probabilities(g, n, m, dev)
        P = XR.view(m, 3, n)
        k = torch.arange(t, device=dev) % m
        causal = 2.0 * P[k, 0] + P[k, 1]
    else:
        X = _dosages(g, n, m, dev, c["nan_snps"])
        causal = X[torch.arange(t, device=dev) % m]
        XR = X
        if r == 2 and inter is None:   # [SNP x sex, SNP]
            XR = torch.empty((2 * m, n), dtype=torch.float32, device=dev)
            for c0 in range(0, m, 8192):
                XR[2 * c0:2 * (c0 + 8192):2] = X[c0:c0 + 8192] * XL[1]
                XR[2 * c0 + 1:2 * (c0 + 8192):2] = X[c0:c0 + 8192]
    Y = _traits(g, XL, causal, t, c["patterns"], c["miss"], c["zipf"], dev)
    return XL, XR, Y, inter


def _mix(c):
    """The sizes of the requests: (individuals, traits, covariates, patterns, first SNP, SNPs) each."""
    rng = np.random.Generator(np.random.PCG64(c["mix"]))
    out = []
    for _ in range(c["requests"]):
        n = int(rng.integers(c["n_lo"], c["n_total"]))
        t = int(round(math.exp(rng.uniform(0.0, math.log(c["t_hi"])))))
        nsnp = int(round(math.exp(rng.uniform(math.log(10000), math.log(c["m_total"])))))
        snp0 = int(rng.integers(0, c["m_total"] - nsnp + 1))
        out.append((n, t, int(rng.integers(3, 7)), min(t, int(rng.integers(1, 5))), snp0, nsnp))
    return out


def _serve_inputs(c, seed):
    dev = torch.device("cuda")
    g = _gen(seed, dev)
    n_total, m_total = c["n_total"], c["m_total"]
    G = _dosages(g, n_total, m_total, dev)
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    reqs = []
    for n, t, l, patterns, snp0, nsnp in _mix(c):
        rows = np.sort(rng.choice(n_total, n, replace=False)).astype(np.int32)
        XL = _covariates(g, n, l, dev)
        causal = G[snp0 + torch.arange(t, device=dev) % nsnp][:, torch.from_numpy(rows).to(dev).long()]
        Y = _traits(g, XL, causal, t, patterns, 0.10, False, dev)
        reqs.append((rows, XL, Y, snp0, nsnp))
    return G, reqs


def _noalloc_inputs(c, seed):
    dev = torch.device("cuda")
    g = _gen(seed, dev)
    XL = _covariates(g, c["n"], c["l"], dev)
    XR = _dosages(g, c["n"], c["m"], dev)
    Y = _traits(g, XL, XR[torch.arange(c["t"], device=dev) % c["m"]], c["t"], 0, c["miss"], False, dev)
    return XL, XR, Y


# ---------------------------------------------------------------------------
# what a user's program has in hand, and one pass
# ---------------------------------------------------------------------------
def _min_t(c):
    return T_NOMINAL if c["store"] == "all" else T_GENOME_WIDE


def prepare(case, seed):
    c = case
    if c["kind"] == "serve":
        G, reqs = _serve_inputs(c, seed)
        cohorts, queue, keep = {}, [], [G]
        for k, (rows, XL, Y, snp0, nsnp) in enumerate(reqs):
            cohorts[k] = S.Cohort(cid=k, rows=rows, XL=XL.cpu().numpy())
            queue.append(S.Request(rid=k, cohort=k, snp0=snp0, nsnp=nsnp, y_ptr=Y.data_ptr(), t=Y.shape[0]))
            keep.append(Y)
        torch.cuda.synchronize()
        srv = S.Server(G.data_ptr(), c["n_total"], c["m_total"], cohorts, budget_bytes=48 << 30,
                       min_p_store=5e-8, reuse_engines=False)
        return {"kind": "serve", "server": srv, "queue": queue, "keep": keep}
    if c["kind"] == "noalloc":
        XL, XR, Y = _noalloc_inputs(c, seed)
        out = [torch.empty((c["t"], c["m"], c["r"]), device=XL.device) for _ in range(3)]
        out.append(torch.empty((c["t"], c["m"]), device=XL.device))
        return {"kind": "noalloc", "case": c, "XL": XL, "XR": XR, "Y": Y, "out": out}
    XL, XR, Y, inter = _scan_inputs(c, seed)
    eng = E.Engine(c["n"], c["l"], c["r"], c["t"], c["m"],
                   precision=E.MIXED if c["precision"] == "mixed" else E.PLAIN, store_all=c["store"] == "all",
                   disp_cov=c["cov"], min_t_store=_min_t(c), min_r2_store=MIN_R2)
    eng.set_covariates(XL.cpu().numpy())
    if c["model"] == "probs":
        eng.set_column_model(3, [2.0, 1.0, 0.0], combine=True)
    elif inter is not None:
        eng.set_interactions(inter.cpu().numpy(), keep=True)
    torch.cuda.synchronize()
    eng.set_traits_device(Y.data_ptr(), c["t"])
    state = {"kind": "scan", "case": c, "engine": eng, "Y": Y, "XR": XR, "host": None}
    if c["source"] == "host":
        pinned = torch.empty(XR.shape, dtype=torch.float32, pin_memory=True)
        pinned.copy_(XR)
        torch.cuda.synchronize()
        state["XR"], state["pinned"], state["host"] = None, pinned, pinned.numpy()
    return state


def _table(rows, capacity):
    """The stored rows (arrays of one length) in tables of `capacity` entries, unused ones zero, with their count."""
    n = rows["trait"].shape[0]
    out = {"rows": n, "tests": rows.pop("tests"), "singular": rows.pop("singular")}
    for k, v in rows.items():
        full = v.new_zeros if isinstance(v, torch.Tensor) else (lambda shape, v=v: np.zeros(shape, v.dtype))
        if n < capacity:
            w = full((capacity,) + tuple(v.shape[1:]))
            w[:n] = v
            v = w
        out[k] = v
    return out


def _capacity(t, m, store_all):
    return t * m if store_all else min(t * m, 2 * t + 64)


def _rows(s, capacity):
    return _table({"trait": s.trait, "snp": s.snp, "r2": s.r2, "n_used": s.n_used, "mask": s.mask.astype(np.int32),
                   "beta": s.B, "se": s.SE, "t": s.T, "tests": s.tests, "singular": s.singular}, capacity)


def run(state):
    if state["kind"] == "serve":
        res = state["server"].run(state["queue"], realtime=False)
        return [_rows(x.rows, _capacity(q.t, q.nsnp, False)) for x, q in zip(res, state["queue"])]
    if state["kind"] == "noalloc":
        c, o = state["case"], state["out"]
        E.scan_dense_noalloc(state["XL"].data_ptr(), state["Y"].data_ptr(), state["XR"].data_ptr(), c["n"], c["l"],
                             c["r"], c["t"], c["m"], o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(),
                             o[3].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"beta": o[0], "se": o[1], "t": o[2], "r2": o[3]}
    c, eng = state["case"], state["engine"]
    if c["new_traits"]:
        eng.set_traits_device(state["Y"].data_ptr(), c["t"])
    room = _capacity(c["t"], c["m"], c["store"] == "all")
    if state["host"] is not None:
        return _rows(eng.run(state["host"]), room)
    return _rows(eng.scan(state["XR"].data_ptr(), c["m"]), room)


def work(case):
    c = case
    if c["kind"] == "serve":
        mix = _mix(c)
        return {"bytes": sum(4.0 * n * (nsnp + t + l) for n, t, l, _, _, nsnp in mix),
                "flops": sum(2.0 * n * nsnp * (t + l + 1) for n, t, l, _, _, nsnp in mix)}
    n, m, t, l, r = c["n"], c["m"], c["t"], c["l"], c["r"]
    in_cols = {"probs": 2, "inter": 1}.get(c.get("model"), r)   # the third probability has no weight
    out = 4.0 * m * t * (3 * r + 1) if c["kind"] == "noalloc" else 0.0
    if c["kind"] == "scan" and c["store"] == "all":
        out = 4.0 * m * t * (5 + 3 * (l + r))
    flops = 2.0 * n * m * r * (t + l) + 1.0 * n * m * r * (r + 1)
    return {"bytes": 4.0 * n * (in_cols * m + t + l) + out, "flops": flops}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits
# ---------------------------------------------------------------------------
def _exact_dense(XL, Y, columns, m, r, cov, chunk):
    """Yields (first SNP, beta, se, t (c, t, p), r2, rss (c, t)) of SNP chunks; columns(c0, c1) -> (c, r, n) float64.

    Least squares of each trait on [XL, x] over its observed rows; standard
    errors from the all-rows inverse scaled by (observed / n), residual
    degrees of freedom observed - p, R2 with (n - 1) and (observed - p - 1).
    """
    dev, f8 = XL.device, torch.float64
    l, n = XL.shape
    t, p = Y.shape[0], l + r
    XL = XL.to(f8)
    seen = ~torch.isnan(Y)
    masks, pat = torch.unique(seen, dim=0, return_inverse=True)
    G = masks.shape[0]
    Qg = torch.zeros((G, l, n), dtype=f8, device=dev)
    Ri = torch.empty((G, l, l), dtype=f8, device=dev)
    for g in range(G):
        q, rr = torch.linalg.qr(XL[:, masks[g]].T)
        Qg[g][:, masks[g]] = q.T
        Ri[g] = torch.linalg.inv(rr)
    y = torch.where(seen, Y.to(f8), torch.zeros((), dtype=f8, device=dev))
    b0 = torch.empty((t, l), dtype=f8, device=dev)
    for g in range(G):
        b0[pat == g] = y[pat == g] @ Qg[g].T
    yt = torch.empty_like(y)
    for g in range(G):
        yt[pat == g] = y[pat == g] - b0[pat == g] @ Qg[g]
    nobs = seen.sum(1).to(f8)
    rss0 = (yt * yt).sum(1)
    sst = (y * y).sum(1) - y.sum(1) ** 2 / nobs
    ncorr = nobs - p
    qa, ra = torch.linalg.qr(XL.T)
    qa = qa.T
    rai = torch.linalg.inv(ra)
    mask8 = masks.to(f8)
    QgF = Qg.reshape(G * l, n)
    inv = (lambda s: 1.0 / s) if r == 1 else torch.linalg.inv
    for c0 in range(0, m, chunk):
        c1 = min(m, c0 + chunk)
        X = columns(c0, c1)
        c = c1 - c0
        bad = torch.isnan(X)
        if bool(bad.any()):
            ok = (~bad).sum(2, keepdim=True)
            mean = torch.where(bad, torch.zeros_like(X), X).sum(2, keepdim=True) / ok
            X = torch.where(bad, mean, X)
        X = X - X.mean(2, keepdim=True)
        flat = X.reshape(c * r, n)
        z = (flat @ yt.T).view(c, r, t).transpose(1, 2)                       # (c, t, r)
        A = (flat @ QgF.T).view(c, r, G, l).permute(0, 2, 3, 1)               # (c, G, l, r)
        D = torch.empty((c, G, r, r), dtype=f8, device=dev)
        for a in range(r):
            for b in range(a + 1):
                D[:, :, a, b] = D[:, :, b, a] = (X[:, a] * X[:, b]) @ mask8.T
        Si = inv(D - A.transpose(2, 3) @ A)                                    # (c, G, r, r)
        Aa = (flat @ qa.T).view(c, r, l).transpose(1, 2)                      # (c, l, r)
        Sa = inv(X @ X.transpose(1, 2) - Aa.transpose(1, 2) @ Aa)
        bx = (Si[:, pat] @ z.unsqueeze(3)).squeeze(3)                         # (c, t, r)
        rss = rss0 - (z * bx).sum(2)
        sig = torch.sqrt(torch.clamp(rss, min=0.0) / ncorr)
        beta = torch.zeros((c, t, p), dtype=f8, device=dev)
        se = torch.zeros_like(beta)
        beta[:, :, l:] = bx
        var = torch.zeros((c, p), dtype=f8, device=dev)
        var[:, l:] = torch.diagonal(Sa, dim1=1, dim2=2)
        if cov:
            fit = b0 - (A[:, pat] @ bx.unsqueeze(3)).squeeze(3)               # (c, t, l) orthonormal basis
            beta[:, :, 1:l] = (Ri[pat] @ fit.unsqueeze(3)).squeeze(3)[:, :, 1:]
            RA = rai @ Aa                                                     # (c, l, r)
            var[:, 1:l] = ((rai * rai).sum(1) + ((RA @ Sa) * RA).sum(2))[:, 1:]
        h0 = 1 if cov else l
        se[:, :, h0:] = sig.unsqueeze(2) * torch.sqrt(var[:, None, h0:] * (nobs / n)[None, :, None])
        tt = torch.zeros_like(beta)
        tt[:, :, h0:] = (beta[:, :, h0:] / se[:, :, h0:]).abs()
        r2 = 1.0 - (rss / (ncorr - 1.0)) / (sst / (n - 1.0))
        yield c0, beta, se, tt, r2, rss


def _exact_rows(XL, Y, columns, m, r, cov, store_all, min_t, chunk):
    l, n = XL.shape
    t = Y.shape[0]
    h0 = 1 if cov else l
    nobs = (~torch.isnan(Y)).sum(1)
    parts = []
    for c0, beta, se, tt, r2, rss in _exact_dense(XL, Y, columns, m, r, cov, chunk):
        keep = (tt > min_t) if not store_all else torch.ones_like(tt, dtype=torch.bool)
        keep[:, :, :h0] = False
        live = (rss > 0) & ((r2 > MIN_R2) | store_all) & keep[:, :, l:].any(2)
        i, j = torch.nonzero(live, as_tuple=True)
        bits = (keep[i, j].int() << torch.arange(l + r, device=keep.device, dtype=torch.int32)).sum(1)
        parts.append((j, i + c0, r2[i, j], bits, beta[i, j], se[i, j], tt[i, j]))
    cat = [torch.cat(x) for x in zip(*parts)]
    order = torch.argsort(cat[0] * m + cat[1])
    trait, snp, r2, bits, beta, se, tt = (x[order] for x in cat)
    return _table({"trait": trait.int(), "snp": snp.int(), "r2": r2, "n_used": nobs[trait].int(), "mask": bits.int(),
                   "beta": beta, "se": se, "t": tt, "tests": m * t, "singular": 0}, _capacity(t, m, store_all))


def _chunk(n, r, t, G):
    # doubles per SNP: its columns a few times, z / beta / se / t, and the sums per pattern
    return max(16, int(4.0e8 / (4 * n * r + 10 * t * (r + 1) + 8 * G * (8 * r + r * r))))


def exact(case, seed):
    c, f8 = case, torch.float64
    if c["kind"] == "serve":
        G, reqs = _serve_inputs(c, seed)
        out = []
        for rows, XL, Y, snp0, nsnp in reqs:
            idx = torch.from_numpy(rows).to(G.device).long()
            cols = lambda a, b: G[snp0 + a:snp0 + b][:, idx].to(f8).unsqueeze(1)  # noqa: E731
            out.append(_exact_rows(XL, Y, cols, nsnp, 1, False, False, 5.451310, _chunk(rows.size, 1, Y.shape[0], 4)))
        return out
    if c["kind"] == "noalloc":
        XL, XR, Y = _noalloc_inputs(c, seed)
        t, m, r = c["t"], c["m"], c["r"]
        out = [torch.empty((t, m, r), dtype=f8, device=XL.device) for _ in range(3)]
        out.append(torch.empty((t, m), dtype=f8, device=XL.device))
        for c0, beta, se, tt, r2, _ in _exact_dense(XL, Y, lambda a, b: XR[a * r:b * r].to(f8).view(b - a, r, -1), m,
                                                    r, False, _chunk(c["n"], r, t, t)):
            s = slice(c0, c0 + beta.shape[0])
            for o, v in zip(out, (beta, se, tt)):
                o[:, s] = v[:, :, c["l"]:].transpose(0, 1)
            out[3][:, s] = r2.T
        return {"beta": out[0], "se": out[1], "t": out[2], "r2": out[3]}
    XL, XR, Y, inter = _scan_inputs(c, seed)
    n, m, r = c["n"], c["m"], c["r"]

    def columns(a, b):
        if c["model"] == "probs":
            P = XR.view(m, 3, n)[a:b].to(f8)
            return (2.0 * P[:, 0] + P[:, 1]).unsqueeze(1)
        if inter is not None:
            x = XR[a:b].to(f8)
            return torch.stack([x * h for h in inter.to(f8)] + [x], dim=1)
        return XR[a * r:b * r].to(f8).view(b - a, r, n)

    G = c["patterns"] or c["t"]
    return _exact_rows(XL, Y, columns, m, r, c["cov"], c["store"] == "all", _min_t(c), _chunk(n, r, c["t"], G))
