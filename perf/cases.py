"""
The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values with a ``kind``; each kind is one public entry point:

* ``scan``      perms.perm_threshold, the call that the CLI makes for a batch of phenotypes: standardise, permute,
                then the LOCO (or single-kinship) scan, in the ``fast`` form (what the drop-in installer binds) or the
                ``plain`` form (the function's own default);
* ``grouped``   groups.perm_threshold_grouped, the same with missing phenotype values: one scan per missingness
                pattern;
* ``wald``      core.snp_wald_scan_compat, one block of variants tested against a spectrum that is kept;
* ``gls``       gls.loco_scan, the scan with the covariates in the model;
* ``gls_wald``  gls.snp_wald_scan, one rotated block against a kept spectrum and fitted deltas;
* ``lowrank``   lowrank.loco_scan_resident, the low-rank scan of a resident genotype matrix (FP32 results);
* ``stream``    lowrank_fast.loco_scan_blocks_fast over int8 dosages in pinned host memory;
* ``epi``       epi.snp_wald_scan_batched, anchors x partners of the epistasis scan (results on the host);
* ``post``      post.neg_log10_pvalue, lambda_gc and perm_threshold_p, what is reported of a finished scan.

Sizes are those of this repository's workloads and tests (150 x 1,500 with 100 permutations; 1,000 x 100,000 with
6,484 phenotypes; missingness groups of 1,057-1,600 samples; 20,000-sample low-rank cohorts) and ragged ones between.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "fast-er-lmm_gb300"))

F64 = torch.float64
SEED_PERM = 19930909  # the seed of the reference's permutations
FIELDS = ("f", "beta", "se", "sfve", "nullh2", "max_F")
# relative lengths of the human autosomes, for uneven chromosomes
CHROM_MB = [248, 242, 198, 190, 181, 171, 159, 145, 138, 134, 135, 133, 114, 107, 102, 90, 83, 80, 59, 64, 47, 51]


def listed() -> list[dict]:
    scan = dict(kind="scan", loco=True, n_grid=64, lo=-10.0, hi=10.0, missing=0.0, even=True)
    return [
        # a first look at a small panel: 16 yeast-like chromosomes, 100 permutations; launches and latency count
        dict(scan, name="scan_fast_small", form="fast", N=150, M=1500, chroms=16, D=3, B=20, perms=100, n_grid=100,
             lo=-5.0, hi=5.0),
        # an ordinary study: uneven chromosomes, missing calls, odd sizes throughout
        dict(scan, name="scan_fast_ragged", form="fast", N=563, M=20011, chroms=22, D=4, B=97, perms=37, missing=0.01,
             even=False),
        # the whole published workload shape: molecular phenotypes in bulk
        dict(scan, name="scan_fast_bulk", form="fast", N=1000, M=100_000, chroms=20, D=5, B=6484, perms=10),
        # the default form on an ordinary study
        dict(scan, name="scan_plain_mid", form="plain", N=600, M=20_000, chroms=10, D=4, B=100, perms=20, even=False),
        # phenotypes missing in four patterns, one scan per pattern
        dict(kind="grouped", name="grouped_fast", form="fast", N=1600, M=6000, chroms=8, D=4, B=24, perms=5,
             patterns=4),
        # one chromosome's variants tested against a spectrum that the program keeps
        dict(kind="wald", name="wald_block", N=1000, M=4096, D=5, P=1100, n_real=100),
        # the scan that keeps the covariates in the model, small
        dict(kind="gls", name="gls_loco", N=300, M=3000, chroms=8, C=5, P=60, n_real=60),
        # and its test of one block against a kept spectrum
        dict(kind="gls_wald", name="gls_wald_block", N=800, M=4000, C=5, P=660, n_real=60),
        # a cohort whose kinship is a marker factor, resident genotypes
        dict(kind="lowrank", name="lowrank_resident", N=2000, k=480, M=6000, chroms=8, D=4, P=176, n_real=16),
        # a large cohort, genotypes streamed from the host in blocks
        dict(kind="stream", name="lowrank_stream", N=20_000, k=1000, M=24_576, chroms=4, D=5, P=220, n_real=20),
        # anchors x partners of an epistasis scan, results read on the host
        dict(kind="epi", name="epi_batch", K=3, N=800, C=6, M=6000, P=330, n_real=30, f32=False),
        # what is reported of a finished scan
        dict(kind="post", name="post_stats", M=100_000, B=64, perms=1000, df2=994),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["scan", "scan", "scan", "grouped", "wald", "gls", "gls_wald", "lowrank", "stream", "epi", "post"])
    if kind == "scan":
        form = rng.choice(["fast", "fast", "plain"])
        N = _log(rng, 100, 1300 if form == "fast" else 700)
        M = _log(rng, 1000, 40_000 if form == "fast" else 15_000)
        perms = _log(rng, 5, 100)
        B = _log(rng, 4, 2000 if form == "fast" else 150)
        B = max(1, min(B, (30_000 if form == "fast" else 3000) // (1 + perms)))
        return dict(kind=kind, form=form, N=N, M=M, chroms=rng.randint(1, 22), D=rng.randint(1, 8), B=B, perms=perms,
                    loco=rng.random() < 0.85, n_grid=64, lo=-10.0, hi=10.0, missing=rng.choice([0.0, 0.02]),
                    even=rng.random() < 0.5)
    if kind == "grouped":
        return dict(kind=kind, form="fast", N=_log(rng, 200, 1600), M=_log(rng, 1000, 10_000), chroms=rng.randint(2, 12),
                    D=rng.randint(1, 6), B=_log(rng, 6, 60), perms=_log(rng, 3, 40), patterns=rng.randint(2, 5))
    if kind == "wald":
        P = _log(rng, 50, 3000)
        return dict(kind=kind, N=_log(rng, 100, 1600), M=_log(rng, 200, 8000), D=rng.randint(1, 8), P=P,
                    n_real=rng.randint(1, P))
    if kind == "gls":
        P = _log(rng, 5, 150)
        return dict(kind=kind, N=_log(rng, 100, 500), M=_log(rng, 500, 6000), chroms=rng.randint(2, 10),
                    C=rng.randint(1, 8), P=P, n_real=rng.randint(1, P))
    if kind == "gls_wald":
        P = _log(rng, 20, 1500)
        return dict(kind=kind, N=_log(rng, 100, 1200), M=_log(rng, 200, 6000), C=rng.randint(1, 12), P=P,
                    n_real=rng.randint(1, P))
    if kind == "lowrank":
        P = _log(rng, 10, 400)
        return dict(kind=kind, N=_log(rng, 600, 3000), k=_log(rng, 100, 500), M=_log(rng, 500, 8000),
                    chroms=rng.randint(2, 8), D=rng.randint(1, 6), P=P, n_real=rng.randint(1, P))
    if kind == "stream":
        P = _log(rng, 20, 400)
        return dict(kind=kind, N=_log(rng, 3000, 20_000), k=_log(rng, 200, 1000), M=_log(rng, 2000, 20_000),
                    chroms=rng.randint(2, 6), D=rng.randint(1, 6), P=P, n_real=rng.randint(1, min(P, 50)))
    if kind == "epi":
        P = _log(rng, 20, 600)
        return dict(kind=kind, K=rng.randint(1, 4), N=_log(rng, 100, 1000), C=rng.randint(2, 12),
                    M=_log(rng, 200, 8000), P=P, n_real=rng.randint(1, min(P, 100)), f32=rng.random() < 0.5)
    return dict(kind="post", M=_log(rng, 1000, 200_000), B=_log(rng, 1, 60), perms=_log(rng, 10, 1000),
                df2=_log(rng, 50, 5000))


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _gen(seed: int, salt: int = 0) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1009 + salt)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=F64)


def _rand(g, *shape, dtype=F64):
    return torch.rand(*shape, generator=g, device="cuda", dtype=dtype)


def _dosages(g, N: int, M: int, maf_lo: float = 0.05) -> torch.Tensor:
    """(N, M) int8 Binomial(2, p) calls, p ~ U[maf_lo, 0.5] per variant."""
    p = maf_lo + (0.5 - maf_lo) * _rand(g, M, dtype=torch.float32)
    a = (_rand(g, N, M, dtype=torch.float32) < p).to(torch.int8)
    return a + (_rand(g, N, M, dtype=torch.float32) < p).to(torch.int8)


def _standard(Z: torch.Tensor) -> torch.Tensor:
    """Columns to mean 0 and population variance 1 over the observed calls, missing calls to 0."""
    ok = ~torch.isnan(Z)
    n = ok.sum(0).clamp(min=1)
    z = torch.where(ok, Z, torch.zeros_like(Z))
    mean = z.sum(0) / n
    d = torch.where(ok, z - mean, torch.zeros_like(z))
    sd = ((d * d).sum(0) / n).sqrt()
    return d / torch.where(sd == 0, torch.full_like(sd, float("inf")), sd)


def _chroms(M: int, n: int, even: bool) -> np.ndarray:
    n = min(n, M)
    w = np.ones(n) if even else np.asarray(CHROM_MB[:n], dtype=np.float64)
    sizes = np.maximum(1, np.floor(M * w / w.sum()).astype(int))
    sizes[0] += M - sizes.sum()
    return np.repeat(np.arange(1, n + 1), sizes)


def _covariates(g, N: int, D: int) -> torch.Tensor:
    return torch.cat([torch.ones(N, 1, device="cuda", dtype=F64), _randn(g, N, D - 1)], dim=1)


def _rank_normal(Y: torch.Tensor) -> torch.Tensor:
    """Blom rank-inverse-normal transform per column, missing values kept."""
    ok = ~torch.isnan(Y)
    n = ok.sum(0)
    r = torch.where(ok, Y, torch.full_like(Y, float("inf"))).argsort(0).argsort(0).to(F64) + 1.0
    q = (r - 0.375) / (n + 0.25)
    out = math.sqrt(2.0) * torch.erfinv(2.0 * q.clamp(1e-9, 1 - 1e-9) - 1.0)
    return torch.where(ok, out, torch.full_like(out, float("nan")))


def _phenotypes(g, Z: torch.Tensor, B: int, k: int = 10, h2_hi: float = 0.9) -> torch.Tensor:
    """(N, B): up to k causal variants each, heritabilities U[0, h2_hi]."""
    N, M = Z.shape
    idx = (_rand(g, k, B) * M).long().clamp(max=M - 1)
    eff = _randn(g, k, B) * (_rand(g, k, B) < 0.7)
    y = torch.zeros(N, B, device="cuda", dtype=F64)
    for j in range(k):
        y += torch.nan_to_num(Z[:, idx[j]].to(F64)) * eff[j]
    y = y - y.mean(0)
    y = y / y.std(0).clamp(min=1e-12)
    h2 = h2_hi * _rand(g, B)
    return y * h2.sqrt() + _randn(g, N, B) * (1 - h2).sqrt()


def _scan_data(c: dict, seed: int) -> SimpleNamespace:
    g = _gen(seed, 1)
    N, M = c["N"], c["M"]
    G = _dosages(g, N, M, 0.01)
    Y = _phenotypes(g, G, c["B"], k=30)
    Z = G.to(F64)
    if c.get("missing"):
        Z[_rand(g, N, M, dtype=torch.float32) < c["missing"]] = float("nan")
    if c["kind"] == "grouped":
        # pattern k lacks a share of the samples, the same count for every seed
        pattern = torch.arange(c["B"], device="cuda") % c["patterns"]
        for k in range(1, c["patterns"]):
            gone = torch.zeros(N, dtype=torch.bool, device="cuda")
            gone[_rand(g, N).argsort()[:int(0.34 * k / c["patterns"] * N)]] = True
            Y[gone[:, None] & (pattern == k)[None, :]] = float("nan")
    return SimpleNamespace(Z=Z, Y=_rank_normal(Y), X=_covariates(g, N, c["D"]),
                           chrom=_chroms(M, c["chroms"], c.get("even", False)), Z_kin=None, chrom_kin=None)


def _compat_block(c: dict, seed: int) -> SimpleNamespace:
    g = _gen(seed, 2)
    N = c["N"]
    Zk = _standard(_dosages(g, N, 2 * N).to(F64))
    S = _standard(_dosages(g, N, c["M"]).to(F64))
    return SimpleNamespace(K=Zk @ Zk.T / Zk.shape[1], X=_covariates(g, N, c["D"]),
                           Y=_rank_normal(_phenotypes(g, S, c["P"])), S=S, ld=-3.0 + 7.0 * _rand(g, c["P"]))


def _gls_block(c: dict, seed: int) -> SimpleNamespace:
    b = _compat_block(dict(c, D=c["C"]), seed)
    ev, U = torch.linalg.eigh(b.K + 1e-6 * torch.eye(c["N"], device="cuda", dtype=F64))
    b.s, b.U = ev.clamp(min=0.0), U
    b.Xr, b.Yr, b.Sr = U.T @ b.X, U.T @ b.Y, U.T @ b.S
    return b


def _gls_data(c: dict, seed: int) -> SimpleNamespace:
    g = _gen(seed, 3)
    Z = _standard(_dosages(g, c["N"], c["M"]).to(F64))
    return SimpleNamespace(Z=Z, X=_covariates(g, c["N"], c["C"]), Y=_rank_normal(_phenotypes(g, Z, c["P"])),
                           chrom=_chroms(c["M"], c["chroms"], False))


def _lowrank_data(c: dict, seed: int) -> SimpleNamespace:
    g = _gen(seed, 4)
    N, M = c["N"], c["M"]
    G = _standard(_dosages(g, N, c["k"]).to(F64))
    D8 = _dosages(g, N, M)
    Y = _rank_normal(_phenotypes(g, D8, c["P"], h2_hi=0.7) + 0.3 * G @ _randn(g, c["k"], c["P"]) / math.sqrt(c["k"]))
    return SimpleNamespace(G=G, D8=D8, X=_covariates(g, N, c["D"]), Y=Y, chrom=_chroms(M, c["chroms"], False),
                           g_chrom=_chroms(c["k"], c["chroms"], False))


def _epi_data(c: dict, seed: int) -> SimpleNamespace:
    g = _gen(seed, 5)
    K, N, C, M, P = c["K"], c["N"], c["C"], c["M"], c["P"]
    s = (-torch.log(_rand(g, N).clamp(min=1e-12))).sort(descending=True).values
    X = _randn(g, 1, N, C).repeat(K, 1, 1)
    X[:, :, -1] = _randn(g, K, N)
    dt = torch.float32 if c["f32"] else F64
    return SimpleNamespace(s=s.to(dt), X=X.to(dt), Y=_randn(g, N, P).to(dt), ld=(-3.0 + 7.0 * _rand(g, P)).to(dt),
                           S=_randn(g, K, N, M).to(dt))


def _post_data(c: dict, seed: int) -> SimpleNamespace:
    g = _gen(seed, 6)
    # F(1, df) statistics under the null, a share of them associated
    t = _randn(g, c["M"], c["B"])
    t = torch.where(_rand(g, c["M"], c["B"]) < 0.01, 4.0 * t, t)
    return SimpleNamespace(F=t * t, pmax=18.0 + 6.0 * _rand(g, c["B"], c["perms"]) ** 2)


def prepare(case: dict, seed: int):
    from fasterlmm_gb300 import core, gls
    kind = case["kind"]
    if kind in ("scan", "grouped"):
        return case, _scan_data(case, seed)
    if kind == "wald":  # the program keeps the spectrum and the fitted deltas
        b = _compat_block(case, seed)
        return case, SimpleNamespace(spec=core.fastlmm_compat_rotate(b.K, b.X, b.Y), ld=b.ld, S=b.S)
    if kind == "gls":
        return case, _gls_data(case, seed)
    if kind == "gls_wald":
        b = _gls_block(case, seed)
        row = lambda t: t.contiguous()
        spec = gls.Spectrum(s=b.s, U=b.U, X_rot=b.Xr, Y_rot=b.Yr, Ut=row(b.U.T), Xrt=row(b.Xr.T), Yrt=row(b.Yr.T))
        return case, SimpleNamespace(spec=spec, ld=b.ld, S=b.Sr)
    if kind == "lowrank":
        d = _lowrank_data(case, seed)
        d.Z = _standard(d.D8.to(F64))
        return case, d
    if kind == "stream":
        d = _lowrank_data(case, seed)
        d.host = torch.empty(case["M"], case["N"], dtype=torch.int8, pin_memory=True)
        d.host.copy_(d.D8.T)
        d.rows_of = {int(k): np.flatnonzero(d.chrom == k) for k in np.unique(d.chrom)}
        del d.D8
        return case, d
    if kind == "epi":
        return case, _epi_data(case, seed)
    return case, _post_data(case, seed)


# ---- one pass -------------------------------------------------------------------------------------------------------

def _fields(res) -> dict:
    return {k: getattr(res, k) for k in FIELDS}


def run(state):
    from fasterlmm_gb300 import core, epi, gls, groups, lowrank, lowrank_fast, perms, post
    c, d = state
    kind = c["kind"]
    if kind == "scan":
        res, pmf = perms.perm_threshold(d, list(range(c["B"])), n_perm=c["perms"], loco=c["loco"], n_grid=c["n_grid"],
                                        log_delta_min=c["lo"], log_delta_max=c["hi"], form=c["form"])
        return dict(_fields(res), perm_max_F=pmf)
    if kind == "grouped":
        out = groups.perm_threshold_grouped(d, list(range(c["B"])), n_perm=c["perms"], form=c["form"])
        return [dict(_fields(r.res), perm_max_F=r.perm_max_F) for r in out]
    if kind == "wald":
        return _fields(core.snp_wald_scan_compat(d.spec, d.ld, d.S, n_real=c["n_real"]))
    if kind == "gls":
        return _fields(gls.loco_scan(d.Z, d.X, d.Y, d.chrom, n_real=c["n_real"]))
    if kind == "gls_wald":
        return _fields(gls.snp_wald_scan(d.spec, d.ld, d.S, n_real=c["n_real"]))
    if kind == "lowrank":
        return _fields(lowrank.loco_scan_resident(d.Z, d.chrom, d.G, d.g_chrom, d.X, d.Y, n_real=c["n_real"]))
    if kind == "stream":
        src = lowrank_fast.dosage_blocks(d.host, d.rows_of, torch.device("cuda", torch.cuda.current_device()))
        return _fields(lowrank_fast.loco_scan_blocks_fast(d.G, d.g_chrom, src, c["M"], sorted(d.rows_of), d.X, d.Y,
                                                          n_real=c["n_real"]))
    if kind == "epi":
        return epi.snp_wald_scan_batched(d.s, d.X, d.Y, d.ld, d.S, n_real=c["n_real"])
    lam, used = post.lambda_gc(d.F, c["df2"])
    return dict(neg_log10_p=post.neg_log10_pvalue(d.F, c["df2"]), lambda_gc=lam, used=used,
                threshold=post.perm_threshold_p(d.pmax, c["df2"]))


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def work(case: dict) -> dict:
    c = case
    kind = c["kind"]
    if kind in ("scan", "grouped"):
        N, M, B, P = c["N"], c["M"], c["B"], c["B"] * (1 + c["perms"])
        units = min(c["chroms"], M) if c.get("loco", True) else 1
        groups_ = c.get("patterns", 1)
        share = 1.0 / groups_  # each pattern scans its own phenotypes
        n = N - c["D"]
        flops = groups_ * (2.0 * N * N * M + units * 6.0 * N ** 3 + 2.0 * N * n * M) \
            + groups_ * share * (units * (2.0 * N * n * P + 2.0 * c.get("n_grid", 64) * n * P) + 4.0 * n * P * M)
        return {"bytes": 8.0 * (N * M + N * (B + c["D"]) + 5.0 * M * B + 2.0 * P), "flops": flops}
    if kind == "wald":
        N, M, P, R = c["N"], c["M"], c["P"], c["n_real"]
        return {"bytes": 8.0 * (N * M + N * N + N * P + 5.0 * M * R + P), "flops": 2.0 * N * N * M + 4.0 * N * P * M}
    if kind == "gls":
        N, M, P, C = c["N"], c["M"], c["P"], c["C"]
        u = c["chroms"]
        return {"bytes": 8.0 * (N * M + N * (P + C) + 5.0 * M * c["n_real"] + P),
                "flops": 4.0 * N * N * M + u * (6.0 * N ** 3 + 2.0 * N * N * (P + C) + (64 + 52) * 2.0 * (C + 1) * N * P)
                + 2.0 * (C + 2) * N * P * M}
    if kind == "gls_wald":
        N, M, P, C = c["N"], c["M"], c["P"], c["C"]
        return {"bytes": 8.0 * (N * (M + P + C) + 5.0 * M * c["n_real"] + P), "flops": 2.0 * (C + 2) * N * P * M}
    if kind in ("lowrank", "stream"):
        N, M, P, k, u = c["N"], c["M"], c["P"], c["k"], c["chroms"]
        size_in, size_out = (8.0, 4.0) if kind == "lowrank" else (1.0, 8.0)
        flops = 2.0 * k * k * N + u * (6.0 * k ** 3 + 2.0 * k * k * N + 4.0 * N * k * P + 2.0 * 64 * k * P) \
            + 4.0 * N * k * M + 4.0 * (N + k) * P * M
        return {"bytes": size_in * N * M + 8.0 * N * (k + P) + size_out * (5.0 * M * c["n_real"] + P), "flops": flops}
    if kind == "epi":
        K, N, C, M, P = c["K"], c["N"], c["C"], c["M"], c["P"]
        e = 4.0 if c["f32"] else 8.0
        return {"bytes": e * (K * N * (C + M) + N * P + 3.0 * K * M * c["n_real"] + K * P) + 8.0 * K * P,
                "flops": 2.0 * K * N * P * M * (C + 2)}
    M, B = c["M"], c["B"]
    # the tail of one statistic: about ten terms of the fraction with a handful of operations each, twice
    return {"bytes": 8.0 * (2.0 * M * B + B * c["perms"]), "flops": 2.0 * 10 * 20.0 * M * B}


# ---- plain 64-bit restatement ---------------------------------------------------------------------------------------

def _project(A, X):
    Q, _ = torch.linalg.qr(X)
    return A - Q @ (Q.T @ A)


def _golden(loss_grid, loss_at, n_grid, lo, hi, chunk):
    """Grid argmin, then 50 golden-section steps between its neighbours, for columns in chunks."""
    grid = torch.linspace(lo, hi, n_grid, dtype=F64, device="cuda")
    phi = 2.0 / (1.0 + math.sqrt(5.0))
    phi2 = phi * phi
    out = []
    for cols in chunk:
        i = loss_grid(grid, cols).argmin(0)
        a, b = grid[(i - 1).clamp(min=0)], grid[(i + 1).clamp(max=n_grid - 1)]
        x, y = a + phi2 * (b - a), a + phi * (b - a)
        fx, fy = loss_at(x, cols), loss_at(y, cols)
        for _ in range(50):
            left = fx < fy
            b, a = torch.where(left, y, b), torch.where(left, a, x)
            x, y = a + phi2 * (b - a), a + phi * (b - a)
            fx, fy = loss_at(x, cols), loss_at(y, cols)
        out.append((0.5 * (a + b)).clamp(lo, hi))
    return torch.cat(out)


def _columns(P: int, N: int):
    step = max(1, 40_000_000 // max(N, 1))
    return [slice(a, min(P, a + step)) for a in range(0, P, step)]


def _fit(s, UY, n_grid, lo, hi, yy=None, neff=None, extra=0.0):
    """ML log delta per column of UY (n, P); yy the off-rank sums of squares, extra the count of log(delta) terms."""
    n = s.shape[0] if neff is None else neff
    yy = torch.zeros(UY.shape[1], dtype=F64, device="cuda") if yy is None else yy
    form = lambda q, sl: n * (math.log(2 * math.pi) + torch.log((q / n).clamp(min=1e-300)) + 1.0) + sl

    def on_grid(grid, cols):
        d = grid.exp()[:, None]
        return form((1.0 / (s[None, :] + d)) @ (UY[:, cols] ** 2) + yy[None, cols] / d,
                    (torch.log(s[None, :] + d).sum(1) + extra * grid)[:, None])

    def at(x, cols):
        d = x.exp()
        sd = s[:, None] + d[None, :]
        return form((UY[:, cols] ** 2 / sd).sum(0) + yy[cols] / d, torch.log(sd).sum(0) + extra * x)

    return _golden(on_grid, at, n_grid, lo, hi, _columns(UY.shape[1], s.shape[0]))


def _wald_into(out, where, num, den, rwr, df, n_real):
    """F, beta, SE, SFVE of (P, m) sums into rows `where` of the outputs, and the columns' maxima."""
    beta = num / den
    q = num * num
    var = ((rwr[:, None] - q / den).clamp(min=1e-300) / df) / den
    F = beta * beta / var
    r = slice(0, n_real)
    out["f"][where], out["beta"][where], out["se"][where] = F[r].T, beta[r].T, var[r].sqrt().T
    out["sfve"][where] = (q[r] / (den[r] * rwr[r, None])).clamp(min=0).sqrt().T
    out["max_F"] = torch.maximum(out["max_F"], F.max(1).values)


def _outputs(M, n_real, P):
    out = {k: torch.zeros(M, n_real, dtype=F64, device="cuda") for k in FIELDS[:5]}
    out["max_F"] = torch.full((P,), -math.inf, dtype=F64, device="cuda")
    return out


def _weighted(s, ld, UY, US, off=None):
    """sWy, sWs (P, m) and rWr (P,) with w = 1 / (s + delta); off = (UUY, UUS) adds their 1 / delta terms."""
    d = ld.exp()
    w = 1.0 / (s[:, None] + d[None, :])
    num, den, rwr = (w * UY).T @ US, w.T @ (US * US), (w * UY * UY).sum(0)
    if off is not None:
        UUY, UUS = off
        num = num + (UUY / d).T @ UUS
        den = den + (UUS * UUS).sum(0)[None, :] / d[:, None]
        rwr = rwr + (UUY * UUY).sum(0) / d
    return num, den.clamp(min=1e-300), rwr.clamp(min=1e-300)


def _scan_exact(c, Z, X, Y, chrom, seed_cols):
    N, M = Z.shape
    B, perms, D = Y.shape[1], c["perms"], X.shape[1]
    Zs = _standard(Z)
    cols = [Y]
    for b in range(B):
        order = np.random.default_rng([SEED_PERM, int(seed_cols[b])]).random((perms, N)).argsort(axis=1)
        cols.append(Y[:, b][torch.from_numpy(order).cuda()].T)
    Ya = torch.cat(cols, dim=1)
    P = Ya.shape[1]
    Yr = _project(Ya, X)
    out = _outputs(M, B, P)
    labels = torch.from_numpy(np.asarray(chrom)).cuda()
    eye = torch.eye(N, dtype=F64, device="cuda")
    for k in (sorted(set(chrom.tolist())) if c.get("loco", True) else [None]):
        here = torch.ones(M, dtype=torch.bool, device="cuda") if k is None else labels == k
        Zk = Zs if k is None else Zs[:, ~here]
        K = Zk @ Zk.T / Zk.shape[1] + eye
        ev, U = torch.linalg.eigh(_project(_project(K, X).T, X))
        s, U = (ev[D:] - 1.0).clamp(min=0.0), U[:, D:]
        UY = U.T @ Yr
        ld = _fit(s, UY, c.get("n_grid", 64), c.get("lo", -10.0), c.get("hi", 10.0))
        rows = torch.nonzero(here).flatten()
        for part in rows.split(max(1, 60_000_000 // P)):
            _wald_into(out, part, *_weighted(s, ld, UY, U.T @ _project(Zs[:, part], X)), N - D - 1, B)
        out["nullh2"][rows] = (1.0 / (1.0 + ld[:B].exp()))[None, :]
    out["perm_max_F"] = out["max_F"][B:].reshape(B, perms)
    return out


def _gls_terms(w, Xr, Yr):
    """Per column: A = X^T W X, its Cholesky factor, u = X^T W y and y^T W y; w (N, P)."""
    A = torch.einsum("np,nc,nd->pcd", w, Xr, Xr)
    L = torch.linalg.cholesky(A)
    u = torch.einsum("np,nc,np->pc", w, Xr, Yr)
    return L, u, (w * Yr * Yr).sum(0)


def _gls_fit(s, Xr, Yr):
    N, P = Yr.shape
    form = lambda r, sl: N * (math.log(2 * math.pi) + torch.log((r / N).clamp(min=1e-300)) + 1.0) + sl

    def at(x, cols):
        sd = s[:, None] + x.exp()[None, :]
        L, u, yy = _gls_terms(1.0 / sd, Xr, Yr[:, cols])
        z = torch.linalg.solve_triangular(L, u[:, :, None], upper=False)[:, :, 0]
        return form(yy - (z * z).sum(1), torch.log(sd).sum(0))

    def on_grid(grid, cols):
        n = Yr[:, cols].shape[1]
        return torch.stack([at(x.expand(n), cols) for x in grid])

    return _golden(on_grid, at, 64, -10.0, 10.0, [slice(0, P)])


def _gls_block_exact(out, where, s, Xr, Yr, Sr, ld, n_real):
    N, C = Xr.shape
    w = 1.0 / (s[:, None] + ld.exp()[None, :])
    L, u, _ = _gls_terms(w, Xr, Yr)
    bx = torch.cholesky_solve(u[:, :, None], L)[:, :, 0]
    r = Yr - Xr @ bx.T
    for part in torch.arange(Sr.shape[1], device="cuda").split(max(1, 60_000_000 // (Yr.shape[1] * C))):
        S = Sr[:, part]
        num = (w * r).T @ S
        Bm = torch.stack([(w * Xr[:, k:k + 1]).T @ S for k in range(C)], dim=1)
        z = torch.linalg.solve_triangular(L, Bm, upper=False)
        den = (w.T @ (S * S) - (z * z).sum(1)).clamp(min=1e-300)
        _wald_into(out, where[part], num, den, (w * r * r).sum(0), N - C - 1, n_real)
    out["nullh2"][where] = (1.0 / (1.0 + ld[:n_real].exp()))[None, :]


def _lowrank_exact(c, d, Z_of):
    N, D, P, M = c["N"], c["D"], c["P"], c["M"]
    out = _outputs(M, c["n_real"], P)
    Yr = _project(d.Y, d.X)
    for k in sorted(set(d.chrom.tolist())):
        G = _project(d.G[:, torch.from_numpy(d.g_chrom != k).cuda()], d.X)
        ev, V = torch.linalg.eigh(G.T @ G)
        sv = ev.clamp(min=0.0).sqrt()
        keep = sv > 1e-10
        U, s = G @ (V[:, keep] / sv[keep]), ev[keep] / G.shape[1]
        UY = U.T @ Yr
        UUY = Yr - U @ UY
        ld = _fit(s, UY, 64, -10.0, 10.0, (UUY * UUY).sum(0), float(N - D), float(N - D - s.shape[0]))
        rows = torch.from_numpy(np.flatnonzero(d.chrom == k)).cuda()
        for part in rows.split(4096):
            S = _project(Z_of(part), d.X)
            US = U.T @ S
            _wald_into(out, part, *_weighted(s, ld, UY, US, (UUY, S - U @ US)), N - D - 1, c["n_real"])
        out["nullh2"][rows] = (1.0 / (1.0 + ld[:c["n_real"]].exp()))[None, :]
    return out


def _epi_exact(c, d):
    s, X, Y, ld, S = (t.to(F64) for t in (d.s, d.X, d.Y, d.ld, d.S))
    K, N, C, M = c["K"], c["N"], c["C"], c["M"]
    outs = []
    for k in range(K):
        w = 1.0 / (s[:, None] + ld.exp()[None, :])
        L, u, _ = _gls_terms(w, X[k], Y)
        r = Y - X[k] @ torch.cholesky_solve(u[:, :, None], L)[:, :, 0].T
        num = (w * r).T @ S[k]
        sws = w.T @ (S[k] * S[k])
        z = torch.linalg.solve_triangular(L, torch.stack([(w * X[k][:, j:j + 1]).T @ S[k] for j in range(C)], 1),
                                          upper=False)
        raw = sws - (z * z).sum(1)
        den = raw.clamp(min=1e-300)
        beta = num / den
        var = (((w * r * r).sum(0)[:, None] - num * num / den).clamp(min=1e-300) / (N - C - 1)) / den
        F = torch.where(raw < 0.01 * sws, torch.zeros_like(raw), beta * beta / var)
        q = slice(0, c["n_real"])
        outs.append((beta[q].T, var[q].sqrt().T, F[q].T, F.max(1).values))
    return (*(torch.stack(t) for t in zip(*outs)), None)


def _log_tail(F, df):
    """log P(F(1, df) > F) by the continued fraction of the incomplete beta function (Abramowitz & Stegun 26.5.8),
    evaluated backwards from a fixed depth."""
    a, b = 0.5 * df, 0.5
    lbeta = math.lgamma(a) + math.lgamma(b) - math.lgamma(a + b)
    x, y = df / (df + F), F / (df + F)
    pre = -a * torch.log1p(F / df) + b * torch.log(y) - lbeta

    def fraction(p, q, z):
        h = torch.ones_like(z)
        for m in range(120, 0, -1):
            odd = -(p + m) * (p + q + m) * z / ((p + 2 * m) * (p + 2 * m + 1))
            even = m * (q - m) * z / ((p + 2 * m - 1) * (p + 2 * m))
            h = 1.0 + even / (1.0 + odd / h)
        return 1.0 / (1.0 - (p + q) * z / ((p + 1) * h))

    direct = pre + torch.log(fraction(a, b, x)) - math.log(a)
    other = torch.log1p(-(pre.exp() * fraction(b, a, y) / b).clamp(max=1.0))
    return torch.where(x < (a + 1) / (a + b + 2), direct, other)


def _post_exact(c, d):
    df = float(c["df2"])
    logp = torch.cat([_log_tail(f, df) for f in d.F.split(8192)])
    # chi-square quantile of the median p: the median of a decreasing function of F is that of the median F's
    lam = []
    mid = d.F.sort(0).values
    n = d.F.shape[0]
    for i in {(n - 1) // 2, n // 2}:
        p = _log_tail(mid[i], df).exp()
        z = torch.special.ndtri(p / 2)
        lam.append(z * z / 0.45493642311957283)
    pm = _log_tail(d.pmax, df).exp()
    return dict(neg_log10_p=-logp / math.log(10.0), lambda_gc=sum(lam) / len(lam), used=None,
                threshold=torch.quantile(pm, 0.05, dim=1))


def exact(case: dict, seed: int):
    c = case
    kind = c["kind"]
    if work(c)["flops"] > 4e12:  # over a few seconds in 64 bits
        return None
    if kind == "scan":
        d = _scan_data(c, seed)
        return _scan_exact(c, d.Z, d.X, d.Y, d.chrom, range(c["B"]))
    if kind == "grouped":
        d = _scan_data(c, seed)
        gone = torch.isnan(d.Y).cpu().numpy()
        groups_ = {}
        for b in range(c["B"]):
            groups_.setdefault(gone[:, b].tobytes(), []).append(b)
        outs = []
        for cols in groups_.values():
            keep = torch.from_numpy(~gone[:, cols[0]]).cuda()
            if int(keep.sum()) - c["D"] - 1 >= 1:
                outs.append(_scan_exact(c, d.Z[keep], d.X[keep], d.Y[keep][:, cols], d.chrom, cols))
        return outs
    if kind == "wald":
        b = _compat_block(c, seed)
        N, D = c["N"], c["D"]
        K = b.K + torch.eye(N, dtype=F64, device="cuda")
        ev, U = torch.linalg.eigh(_project(_project(K, b.X).T, b.X))
        s, U = (ev[D:] - 1.0).clamp(min=0.0), U[:, D:]
        out = _outputs(c["M"], c["n_real"], c["P"])
        UY = U.T @ _project(b.Y, b.X)
        for part in torch.arange(c["M"], device="cuda").split(max(1, 60_000_000 // c["P"])):
            _wald_into(out, part, *_weighted(s, b.ld, UY, U.T @ _project(b.S[:, part], b.X)), N - D - 1, c["n_real"])
        out["nullh2"][:] = (1.0 / (1.0 + b.ld[:c["n_real"]].exp()))[None, :]
        return out
    if kind == "gls":
        d = _gls_data(c, seed)
        out = _outputs(c["M"], c["n_real"], c["P"])
        labels = torch.from_numpy(d.chrom).cuda()
        for k in sorted(set(d.chrom.tolist())):
            Zk = d.Z[:, labels != k]
            ev, U = torch.linalg.eigh(Zk @ Zk.T / Zk.shape[1] + 1e-6 * torch.eye(c["N"], dtype=F64, device="cuda"))
            s, Xr, Yr = ev.clamp(min=0.0), U.T @ d.X, U.T @ d.Y
            rows = torch.nonzero(labels == k).flatten()
            _gls_block_exact(out, rows, s, Xr, Yr, U.T @ d.Z[:, rows], _gls_fit(s, Xr, Yr), c["n_real"])
        return out
    if kind == "gls_wald":
        b = _gls_block(c, seed)
        out = _outputs(c["M"], c["n_real"], c["P"])
        _gls_block_exact(out, torch.arange(c["M"], device="cuda"), b.s, b.Xr, b.Yr, b.Sr, b.ld, c["n_real"])
        return out
    if kind in ("lowrank", "stream"):
        d = _lowrank_data(c, seed)
        return _lowrank_exact(c, d, lambda rows: _standard(d.D8[:, rows].to(F64)))
    if kind == "epi":
        return _epi_exact(c, _epi_data(c, seed))
    return _post_exact(c, _post_data(c, seed))
