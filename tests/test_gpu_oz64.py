"""
FP64 products on the tensor cores (csrc/flmm_oz64.cu) against exact sums and against the FP64-pipe kernel.

The digit planes must lose no more than an FP64 sum does: over sampled outputs the rms error against exact sums (exact
products by Dekker's splitting, exact addition by math.fsum) is at most that of flmm_gemm_nt_f64.  Rows that digits
cannot hold (not finite, exponents out of range, one entry far above the rest) take the FP64 pipe, bit for bit.
"""
from __future__ import annotations

import math
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _products(A, B, D=None):
    from fasterlmm_gb300 import _lib, build
    from fasterlmm_gb300.core import _ptr, _stream, _work
    build()
    Mr, K = A.shape
    Nr = B.shape[0]
    dev = A.device
    tc = torch.full((Mr, Nr), 7.0, dtype=torch.float64, device=dev)
    ref = torch.empty((Mr, Nr), dtype=torch.float64, device=dev)
    w, wb = _work.get(dev, _lib.query_bytes("flmm_gemm_nt_f64_tc_workspace_bytes", Mr, Nr, K))
    _lib.call("flmm_gemm_nt_f64_tc", _ptr(A), A.stride(0), _ptr(B), B.stride(0), _ptr(D), 0 if D is None else Nr,
              _ptr(tc), Nr, Mr, Nr, K, w, wb, _stream(dev))
    _lib.call("flmm_gemm_nt_f64", _ptr(A), A.stride(0), _ptr(B), B.stride(0), _ptr(ref), Nr, Mr, Nr, K, 1.0, _stream(dev))
    _lib.call("flmm_context_check", _lib.context(dev.index), _stream(dev))
    return tc, ref


def _exact(a, b):
    """Correctly rounded sum of a[k] b[k]."""
    split = lambda x: (lambda c: (c - (c - x), x - (c - (c - x))))(134217729.0 * x)
    (ah, al), (bh, bl) = split(a), split(b)
    p = a * b
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    return math.fsum(np.concatenate([p, e]))


def _rms(x):
    return float(np.sqrt(np.mean(np.square(x))))


@pytest.mark.parametrize("Mr,Nr,K", [(1, 1, 32), (127, 63, 33), (128, 64, 512), (129, 65, 513), (257, 200, 1000),
                                     (300, 130, 1537), (40, 70, 5003)])
@pytest.mark.parametrize("kind", ["normal", "positive"])
def test_no_less_exact_than_fp64(Mr, Nr, K, kind):
    g = torch.Generator(device="cuda").manual_seed(Mr * 7 + K)
    A = torch.randn(Mr, K, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(Nr, K, generator=g, device="cuda", dtype=torch.float64) * 3.0
    if kind == "positive":  # weights and squares, rows of different sizes
        A = 1.0 / (A.abs() + 0.3) * torch.logspace(-20, 20, Mr, device="cuda", dtype=torch.float64)[:, None]
        B = B * B
    tc, ref = _products(A, B)
    a, b, tc, ref = (t.cpu().numpy() for t in (A, B, tc, ref))
    rng = np.random.default_rng(0)
    at = {(0, 0), (Mr - 1, Nr - 1)} | {(int(rng.integers(Mr)), int(rng.integers(Nr))) for _ in range(300)}
    scale = lambda i, j: np.linalg.norm(a[i]) * np.linalg.norm(b[j])
    ex = {ij: _exact(a[ij[0]], b[ij[1]]) for ij in at}
    err = lambda c: _rms([(c[ij] - ex[ij]) / scale(*ij) for ij in at])
    assert err(tc) <= max(err(ref), 2.0 ** -53)


def test_difference_form():
    g = torch.Generator(device="cuda").manual_seed(5)
    A, B = (torch.randn(n, 300, generator=g, device="cuda", dtype=torch.float64) for n in (150, 90))
    D = torch.randn(150, 90, generator=g, device="cuda", dtype=torch.float64)
    tc, _ = _products(A, B)
    dif, _ = _products(A, B, D)
    assert torch.equal(dif, D - tc)


def test_rows_that_digits_cannot_hold():
    """Only the tiles of such rows change path, and there the bits are the FP64 pipe's."""
    g = torch.Generator(device="cuda").manual_seed(6)
    Mr, Nr, K = 400, 200, 600
    A = torch.randn(Mr, K, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(Nr, K, generator=g, device="cuda", dtype=torch.float64)
    A[130, 7] = float("nan")
    A[131, 8] = float("inf")
    A[140] *= 1e200
    A[150, 3] = 1e9      # one entry far above the rest of its row
    A[160] = 0.0
    B[70] *= 1e-200
    tc, ref = _products(A, B)
    bad = torch.zeros(Mr, Nr, dtype=torch.bool, device="cuda")
    bad[128:256] = True
    bad[:, 64:128] = True
    assert torch.equal(torch.isnan(tc), torch.isnan(ref))
    same = (tc == ref) | (torch.isnan(tc) & torch.isnan(ref))
    assert bool(same[bad].all())
    torch.testing.assert_close(tc[~bad], ref[~bad], rtol=0, atol=1e-11)
    assert not same[~bad].all()  # the other tiles ran on the tensor cores


@pytest.mark.parametrize("P,Mc,Neff,n_real", [(40, 300, 130, 40), (129, 1000, 700, 1), (2049, 300, 100, 2049),
                                              (100, 4097, 150, 33), (64, 4160, 257, 1)])
def test_wald_blocks(P, Mc, Neff, n_real):
    """flmm_wald_f64 over its blocks of columns and variants, on either path, against the formulas in FP64."""
    from fasterlmm_gb300 import build, core
    build()
    g = torch.Generator(device="cuda").manual_seed(P + Mc)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    s, UY, US = rn(Neff).abs() + 0.05, rn(P, Neff), rn(Mc, Neff)
    ld = rn(P)
    US[5] = 0.0
    out, max_F = core._alloc_outputs(Mc, n_real, P, dev)
    rows = torch.randperm(Mc, generator=g, device=dev)
    core.wald_t(s, UY, ld, US, n_real, rows, out, max_F)
    w = 1.0 / (s[None, :] + ld.exp()[:, None])
    num, den, rwr = (w * UY) @ US.T, (w @ (US * US).T).clamp(min=1e-300), (w * UY * UY).sum(1)
    var = (rwr[:, None] - num * num / den).clamp(min=1e-300) / (Neff - 1) / den
    F = (num / den) ** 2 / var
    close = lambda x, y: torch.testing.assert_close(x, y, rtol=1e-9, atol=1e-12)
    close(max_F, F.max(1).values)
    r = slice(0, n_real)
    close(out["f"][rows], F[r].T)
    close(out["beta"][rows], (num / den)[r].T)
    close(out["se"][rows], var[r].sqrt().T)
    close(out["sfve"][rows], (num * num / (den * rwr[:, None]))[r].sqrt().T)


def test_wald_keeps_nan():
    from fasterlmm_gb300 import build, core
    build()
    g = torch.Generator(device="cuda").manual_seed(3)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    P, Mc, Neff = 200, 600, 300
    UY = rn(P, Neff)
    UY[3, 5] = UY[150, 2] = float("nan")
    out, max_F = core._alloc_outputs(Mc, 10, P, dev)
    core.wald_t(rn(Neff).abs(), UY, rn(P), rn(Mc, Neff), 10, torch.arange(Mc, device=dev), out, max_F)
    nan = torch.zeros(P, dtype=torch.bool, device=dev)
    nan[3] = nan[150] = True
    assert torch.equal(torch.isnan(max_F), nan)
    assert torch.equal(torch.isnan(out["f"]).any(0), nan[:10])


@pytest.mark.parametrize("P,Mc,N,C,n_real", [(3, 40, 50, 1, 3), (70, 300, 333, 5, 70), (130, 257, 500, 12, 1),
                                             (900, 4100, 120, 5, 17), (40, 600, 400, 30, 40)])
def test_gls_wald_blocks(P, Mc, N, C, n_real):
    """flmm_wald_gls_f64 over its blocks, on either path, against the formulas in FP64."""
    from fasterlmm_gb300 import build, core, gls
    build()
    g = torch.Generator(device="cuda").manual_seed(P + Mc + C)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    s, X, Y, S, ld = rn(N).abs() + 0.05, rn(C, N), rn(P, N), rn(Mc, N), rn(P)
    out, max_F = core._alloc_outputs(Mc, n_real, P, dev)
    rows = torch.randperm(Mc, generator=g, device=dev)
    gls.wald_t(s, X, Y, ld, S, n_real, rows, out, max_F)
    w = 1.0 / (s[None, :] + ld.exp()[:, None])
    L = torch.linalg.cholesky(torch.einsum("pn,cn,dn->pcd", w, X, X))
    u = torch.einsum("pn,cn,pn->pc", w, X, Y)
    r = Y - torch.cholesky_solve(u[:, :, None], L)[:, :, 0] @ X
    z = torch.linalg.solve_triangular(L, torch.einsum("pn,cn,mn->pcm", w, X, S), upper=False)
    num, den, rwr = (w * r) @ S.T, (w @ (S * S).T) - (z * z).sum(1), (w * r * r).sum(1)
    var = (rwr[:, None] - num * num / den) / (N - C - 1) / den
    F = (num / den) ** 2 / var
    close = lambda x, y: torch.testing.assert_close(x, y, rtol=1e-9, atol=1e-12)
    close(max_F, F.max(1).values)
    q = slice(0, n_real)
    close(out["f"][rows], F[q].T)
    close(out["beta"][rows], (num / den)[q].T)
    close(out["se"][rows], var[q].sqrt().T)
    close(out["sfve"][rows], (num * num / (den * rwr[:, None]))[q].sqrt().T)


def test_weights_that_meet_zeros():
    """A direction whose weight is 2e4 times the others' and where every variant is 0 (the rotated intercept at a small
    delta) must not cost the other directions their digits: SE, which is a sum of w s^2, keeps FP64's exactness."""
    from fasterlmm_gb300 import build, core
    build()
    g = torch.Generator(device="cuda").manual_seed(9)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    P, Mc, Neff = 130, 700, 400
    s, UY, US, ld = rn(Neff).abs() + 1.0, rn(P, Neff), rn(Mc, Neff), torch.full((P,), -10.0, device=dev, dtype=torch.float64)
    s[0], UY[:, 0], US[:, 0] = 0.0, 0.0, 0.0
    out, max_F = core._alloc_outputs(Mc, P, P, dev)
    core.wald_t(s, UY, ld, US, P, torch.arange(Mc, device=dev), out, max_F)
    w = 1.0 / (s[None, :] + ld.exp()[:, None])
    num, den, rwr = (w * UY) @ US.T, w @ (US * US).T, (w * UY * UY).sum(1)
    se = ((rwr[:, None] - num * num / den) / (Neff - 1) / den).sqrt()
    torch.testing.assert_close(out["se"], se.T, rtol=1e-14, atol=0)


def _one_entry_scan(entry, K, M, P, C, bad_at, bad_k):
    """beta / se (M, P) with the covariates projected out (C = 0) or in the model, variant bad_at[0] holding `entry` at
    bad_k, and the same in the formulas."""
    from fasterlmm_gb300 import build, core, gls
    build()
    g = torch.Generator(device="cuda").manual_seed(K + C)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    s, Y, S, ld, X = rn(K).abs() + 0.05, rn(P, K), rn(M, K), rn(P), rn(max(C, 1), K)
    if entry is not None:
        S[bad_at, bad_k] = entry
    out, max_F = core._alloc_outputs(M, P, P, dev)
    rows = torch.arange(M, device=dev)
    w = 1.0 / (s[None, :] + ld.exp()[:, None])
    if C:
        gls.wald_t(s, X, Y, ld, S, P, rows, out, max_F)
        L = torch.linalg.cholesky(torch.einsum("pn,cn,dn->pcd", w, X, X))
        u = torch.einsum("pn,cn,pn->pc", w, X, Y)
        r = Y - torch.cholesky_solve(u[:, :, None], L)[:, :, 0] @ X
        z = torch.linalg.solve_triangular(L, torch.einsum("pn,cn,mn->pcm", w, X, S), upper=False)
        num, den, rwr, df = (w * r) @ S.T, (w @ (S * S).T) - (z * z).sum(1), (w * r * r).sum(1), K - C - 1
    else:
        core.wald_t(s, Y, ld, S, P, rows, out, max_F)
        num, den, rwr, df = (w * Y) @ S.T, w @ (S * S).T, (w * Y * Y).sum(1), K - 1
    t = num / ((rwr[:, None] - num * num / den) / df * den).sqrt()
    return out["beta"] / out["se"], t.T, max_F


@pytest.mark.parametrize("entry", [float("nan"), float("inf"), -float("inf"), 1e12, 1e6, 1e3])
@pytest.mark.parametrize("K,C", [(160, 0), (800, 0), (160, 5), (800, 5)])
def test_one_entry_of_one_variant(entry, K, C):
    """A variant that is not finite, or far off, at one index costs the other variants nothing: their statistic
    t = beta / se is what an FP64 sum of K terms allows.  The sums' rounding is at most K 2^-53 of the row norms on either
    side, and t = sWy / sqrt(sWs rss / df) takes it times sqrt(df), once for sWy and at |t| / sqrt(df) < 1 for the others."""
    P, M, at = 260, 700, 333
    t, ref, max_F = _one_entry_scan(entry, K, M, P, C, at, K // 3)
    others = torch.ones(M, dtype=torch.bool, device=t.device)
    others[at] = False
    atol = 8 * K ** 0.5 * K * 2.0 ** -53
    torch.testing.assert_close(t[others], ref[others], rtol=0, atol=atol)
    if abs(entry) < 1e4:  # (further off, one term of the variant's sums is nearly all there is of rss)
        torch.testing.assert_close(t[at], ref[at], rtol=0, atol=64 * atol)
    finite = torch.full_like(max_F, abs(entry) < float("inf"), dtype=torch.bool)
    assert torch.equal(torch.isfinite(t[at]), finite)
    assert torch.equal(torch.isfinite(max_F), finite)


def _loss_of_digits(a, b):
    """rms error of a product of rows a and b from the method, over the row norms: the rounding of both to 55 bits, the
    plane pairs of level 8 (seven, of uniform digits), and the rounding of the result at its own size."""
    na, nb = np.linalg.norm(a), np.linalg.norm(b)
    ea, eb = (2.0 ** np.frexp(np.abs(x).max())[1] for x in (a, b))
    digits = 2.0 ** -56 / 3 ** 0.5 * np.hypot(ea / na, eb / nb)
    level = 2.0 ** -56 * ea * eb / (na * nb) * (7 * a.size) ** 0.5 * (37.0 ** 2 / 2 ** 12)
    return np.sqrt(digits ** 2 + level ** 2 + (2.0 ** -53 / 3 ** 0.5 * abs(a @ b) / (na * nb)) ** 2)


@pytest.mark.parametrize("K", [48, 160, 400, 1000, 2500])
def test_products_no_further_off_than_sums(K):
    """Against exact sums: no further off than the FP64 pipe's chains, or, where those are short, than the method's own loss
    (1.5: the spread of an rms over 300 samples and digits that are not quite uniform)."""
    g = torch.Generator(device="cuda").manual_seed(K)
    A, B = (torch.randn(n, K, generator=g, device="cuda", dtype=torch.float64) for n in (200, 2600))
    tc, ref = _products(A, B)
    a, b, tc, ref = (t.cpu().numpy() for t in (A, B, tc, ref))
    rng = np.random.default_rng(1)
    at = [(int(rng.integers(200)), int(rng.integers(2600))) for _ in range(300)]
    scale = lambda i, j: np.linalg.norm(a[i]) * np.linalg.norm(b[j])
    ex = {ij: _exact(a[ij[0]], b[ij[1]]) for ij in at}
    err = lambda c: _rms([(c[ij] - ex[ij]) / scale(*ij) for ij in at])
    loss = _rms([_loss_of_digits(a[i], b[j]) for i, j in at])
    assert err(tc) <= (err(ref) if K >= 400 else max(err(ref), 1.5 * loss))
    assert err(tc) <= 1.5 * loss


NO_PAIRS = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import torch
from fasterlmm_gb300 import _lib, core
from test_gpu_oz64 import _one_entry_scan, _products
from fasterlmm_gb300.core import _ptr, _stream, _work
g = torch.Generator(device="cuda").manual_seed(4)
A, B, D = (torch.randn(*s, generator=g, device="cuda", dtype=torch.float64) for s in ((300, 200), (400, 200), (300, 400)))
tc, ref = _products(A, B)
assert torch.equal(tc, ref)
want, _ = _products(A, B, D)
torch.testing.assert_close(want, D - ref, rtol=0, atol=1e-12)
w, wb = _work.get(A.device, _lib.query_bytes("flmm_gemm_nt_f64_tc_workspace_bytes", 300, 400, 200))
_lib.call("flmm_gemm_nt_f64_tc", _ptr(A), 200, _ptr(B), 200, _ptr(D), 400, _ptr(D), 400, 300, 400, 200, w, wb, _stream(A.device))
assert torch.equal(D, want)
for C in (0, 3):
    t, ref, _ = _one_entry_scan(None, 200, 600, 200, C, 0, 0)
    torch.testing.assert_close(t, ref, rtol=0, atol=8 * 200 ** 1.5 * 2.0 ** -53)
print("formed on the FP64 pipe")
"""


def test_without_the_tensor_cores():
    """Every tile on the FP64 pipe, as after a wait that k_oz64 gave up: FLMM_TC_PAIR=0 keeps CTA pairs out of the process."""
    tests = Path(__file__).resolve().parent
    code = NO_PAIRS.format(root=str(tests.parent / "fast-er-lmm_gb300"), tests=str(tests))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, FLMM_TC_PAIR="0"), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "formed on the FP64 pipe" in r.stdout, r.stderr[-2000:]


def _wald_call(kind, P, Mc, K, C):
    """(call(work_bytes) -> outputs, full, least): flmm_wald_f64, flmm_wald_gls_f64 or flmm_wald_lowrank_f64 on one problem,
    the workspace that it asks for and the shortest that it takes."""
    from fasterlmm_gb300 import _lib, build, core
    from fasterlmm_gb300.core import _ptr, _stream
    build()
    g = torch.Generator(device="cuda").manual_seed(P + K)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    k = K // 4  # on-rank directions of the low-rank form
    s, X, Y, S, ld = rn(K).abs() + 0.05, rn(C, K), rn(P, K), rn(Mc, K), rn(P)
    Yk, Yn, Sk, Sn = (t.contiguous() for t in (Y[:, :k], Y[:, k:], S[:, :k], S[:, k:]))
    rows = torch.arange(Mc, device=dev)
    cat = 8 * K * (1 + P + Mc) + 256
    query, least = {
        "compat": (("flmm_wald_f64_workspace_bytes", P, K), 8 * (2 * P * K + P) + 512),
        "gls": (("flmm_wald_gls_workspace_bytes", K, C, P), 8 * P * ((C + 2) * K + C * C + 1) + 1024),
        "lowrank": (("flmm_wald_lowrank_f64_workspace_bytes", k, K - k, P, Mc), cat + 8 * (2 * P * K + P) + 512)}[kind]

    def call(nbytes):
        out, max_F = core._alloc_outputs(Mc, P, P, dev)
        work = torch.empty(nbytes + 4096, dtype=torch.uint8, device=dev)
        work[nbytes:] = 171
        o = [_ptr(out[x]) for x in ("f", "beta", "se", "sfve")]
        end = (*o, P, _ptr(max_F), _ptr(work), nbytes, _stream(dev))
        if kind == "compat":
            _lib.call("flmm_wald_f64", _ptr(s), K, _ptr(Y), K, _ptr(ld), P, P, _ptr(S), K, Mc, _ptr(rows), *end)
        elif kind == "gls":
            _lib.call("flmm_wald_gls_f64", _ptr(s), K, _ptr(X), K, C, _ptr(Y), K, _ptr(ld), P, P, _ptr(S), K, Mc, _ptr(rows),
                      *end)
        else:
            _lib.call("flmm_wald_lowrank_f64", _ptr(s), k, _ptr(Yk), k, _ptr(Yn), K - k, K - k, K, _ptr(ld), P, P, _ptr(Sk),
                      k, _ptr(Sn), K - k, Mc, _ptr(rows), *end)
        assert bool((work[nbytes:] == 171).all())  # nothing behind it was written
        return [out[x] for x in ("f", "beta", "se", "sfve")] + [max_F]

    return call, _lib.query_bytes(*query), least


@pytest.mark.parametrize("kind", ["compat", "gls", "lowrank"])
@pytest.mark.parametrize("P,Mc,K,C", [(300, 1500, 400, 5), (129, 4160, 130, 2), (7, 90, 64, 3)])
def test_shorter_workspaces(kind, P, Mc, K, C):
    """Whatever the workspace between the shortest and the one asked for, the same results to the rounding of the sums."""
    from fasterlmm_gb300 import _lib
    call, full, least = _wald_call(kind, P, Mc, K, C)
    want = call(max(full, least))
    for share in (0.0, 0.01, 0.03, 0.1, 0.2, 0.4, 0.7, 1.0):
        for got, ref in zip(call(least + int(share * max(0, full - least))), want):
            torch.testing.assert_close(got, ref, rtol=1e-9, atol=1e-12)
    with pytest.raises(_lib.FlmmError) as e:
        call(min(full, least) - 8)
    assert e.value.status == 4
