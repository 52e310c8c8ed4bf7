"""
The golden-section delta fits with one block per column, at the edges of their chunks of eigenvalues and of the column
counts, against the same search in torch FP64: the losses at the two answers agree to their own rounding (sums of ~n
terms of order 1..10: n 2^-53 relative).
"""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
LO, HI, G = -10.0, 10.0, 64


def _golden(loss, P, dev):
    grid = torch.linspace(LO, HI, G, dtype=torch.float64, device=dev)
    i = torch.stack([loss(x.expand(P)) for x in grid]).argmin(0)
    a, b = grid[(i - 1).clamp(min=0)], grid[(i + 1).clamp(max=G - 1)]
    phi = 2.0 / (1.0 + math.sqrt(5.0))
    for _ in range(50):
        c, d = a + phi * phi * (b - a), a + phi * (b - a)
        left = loss(c) < loss(d)
        b, a = torch.where(left, d, b), torch.where(left, a, c)
    return (0.5 * (a + b)).clamp(LO, HI), i


def _inputs(n, P, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    s = rn(n).abs() * 2
    h2 = torch.rand(P, generator=g, device=dev, dtype=torch.float64)[:, None]
    return s, rn(P, n) * (h2 * s[None, :] + (1 - h2)).sqrt(), rn


@pytest.mark.parametrize("n,P", [(5, 1), (31, 3), (1023, 2), (1024, 5), (1025, 2), (2049, 3), (200, 700)])
def test_compat_fit(n, P):
    from fasterlmm_gb300 import build, core
    build()
    s, UY, _ = _inputs(n, P, n + P)
    ld, idx = core.fit_delta_t(s, UY)

    def loss(x):
        sd = s[None, :] + x.exp()[:, None]
        return n * (math.log(2 * math.pi) + torch.log((UY * UY / sd).sum(1) / n) + 1.0) + torch.log(sd).sum(1)

    want, i = _golden(loss, P, s.device)
    assert torch.equal(idx.long(), i)
    torch.testing.assert_close(loss(ld), loss(want), rtol=n * 2.0 ** -53, atol=1e-11)
    coarse, _ = core.fit_delta_t(s, UY, refine=False)
    assert torch.equal(coarse, torch.linspace(LO, HI, G, dtype=torch.float64, device=s.device)[i])


@pytest.mark.parametrize("n,C,P", [(40, 1, 1), (257, 5, 9), (1025, 3, 2), (120, 30, 3)])
@pytest.mark.parametrize("reml", [False, True])
def test_gls_fit(n, C, P, reml):
    from fasterlmm_gb300 import build, gls
    build()
    s, Y, rn = _inputs(n, P, n + C)
    X = rn(C, n)
    ld, idx = gls.fit_delta_t(s, X, Y, reml=reml)

    def loss(x):
        sd = s[None, :] + x.exp()[:, None]
        w = 1.0 / sd
        L = torch.linalg.cholesky(torch.einsum("pn,cn,dn->pcd", w, X, X))
        z = torch.linalg.solve_triangular(L, torch.einsum("pn,cn,pn->pc", w, X, Y)[:, :, None], upper=False)[:, :, 0]
        rwr = (w * Y * Y).sum(1) - (z * z).sum(1)
        m = n - C if reml else n
        out = m * (math.log(2 * math.pi) + torch.log(rwr / m) + 1.0) + torch.log(sd).sum(1)
        return out + 2 * torch.log(torch.diagonal(L, dim1=1, dim2=2)).sum(1) if reml else out

    want, i = _golden(loss, P, s.device)
    assert torch.equal(idx.long(), i)
    torch.testing.assert_close(loss(ld), loss(want), rtol=4 * n * 2.0 ** -53, atol=1e-10)


@pytest.mark.parametrize("n,P,scale", [(1, 2, 1.0), (33, 40, 1.0), (511, 9, 1.0), (512, 9, 1e-9), (513, 9, 1e5),
                                       (1537, 5, 1.0)])
@pytest.mark.parametrize("off", [0, 7])
def test_steps_taken_from_grouped_sums(n, P, scale, off):
    """The steps that grouped sums decide (groups of 16 x 32 eigenvalues) are the reference's: the answer lies in the bracket
    that the search in torch FP64 has while its two losses still differ by more than 1e-8 (rounding there is ~1e-11)."""
    from fasterlmm_gb300 import build, core, lowrank
    build()
    s, UY, rn = _inputs(n, P, 3 * n + off)
    s = s * scale
    N = n + off
    rest = rn(P, 1 + off)
    yy = rest.square().sum(1)
    if off:
        ld, i = lowrank.fit_delta_t(s, UY, rest, N)
    else:
        ld, i = core.fit_delta_t(s, UY)

    def loss(x):
        sd = s[None, :] + x.exp()[:, None]
        q = (UY * UY / sd).sum(1) + (yy / x.exp() if off else 0.0)
        return N * (math.log(2 * math.pi) + torch.log(q / N) + 1.0) + torch.log(sd).sum(1) + off * x

    grid = torch.linspace(LO, HI, G, dtype=torch.float64, device=s.device)
    i = i.long()  # (eigenvalues of 1e-9 leave the loss flat: the node is rounding's choice)
    a, b = grid[(i - 1).clamp(min=0)], grid[(i + 1).clamp(max=G - 1)]
    phi = 2.0 / (1.0 + math.sqrt(5.0))
    sure = torch.ones(P, dtype=torch.bool, device=s.device)
    for _ in range(50):
        c, d = a + phi * phi * (b - a), a + phi * (b - a)
        fc, fd = loss(c), loss(d)
        sure &= (fc - fd).abs() > 1e-8
        left = fc < fd
        b, a = torch.where(sure & left, d, b), torch.where(sure & ~left, c, a)
    assert ((ld >= a - 1e-12) & (ld <= b + 1e-12)).all()


SPECTRA = {
    "half-normal": lambda g, n: torch.randn(n, generator=g, device="cuda", dtype=torch.float64).abs() * 2,
    "falling": lambda g, n: torch.logspace(2, -9, n, device="cuda", dtype=torch.float64),
    "with zeros": lambda g, n: torch.rand(n, generator=g, device="cuda", dtype=torch.float64).round(decimals=1),
    "one value": lambda g, n: torch.full((n,), 0.75, device="cuda", dtype=torch.float64),
    "tiny": lambda g, n: torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 1e-9,
    "large": lambda g, n: torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 1e5,
}


@pytest.mark.parametrize("spectrum", list(SPECTRA))
@pytest.mark.parametrize("n", [1, 2, 33, 300, 512, 995, 2049])
@pytest.mark.parametrize("off", [0, 7])
def test_certain_steps_leave_every_bit(spectrum, n, off):
    """The search from the list of certain steps ends where the one that evaluates every loss ends, to the bit."""
    from fasterlmm_gb300 import _lib, build
    from fasterlmm_gb300.core import _ptr, _stream
    build()
    g = torch.Generator(device="cuda").manual_seed(n)
    dev = torch.device("cuda", torch.cuda.current_device())
    rn = lambda *x: torch.randn(*x, generator=g, device=dev, dtype=torch.float64)
    s, P = SPECTRA[spectrum](g, n), 240
    h2 = torch.rand(P, generator=g, device=dev, dtype=torch.float64)[:, None]
    UY = rn(P, n) * (h2 * s[None, :] / s.mean() + (1 - h2)).sqrt()
    UY *= torch.logspace(-4, 4, P, device=dev, dtype=torch.float64)[:, None]
    UY[3] = 0.0
    yy = UY.square().sum(1) * rn(P).square() * 0.1 if off else None
    if off:
        yy[5] = 0.0
    got = []
    for refine in (1, 2):
        for lo, hi in ((-10.0, 10.0), (-3.0, 2.5)):
            ld, idx = torch.empty(P, dtype=torch.float64, device=dev), torch.empty(P, dtype=torch.int32, device=dev)
            nbytes = _lib.query_bytes("flmm_fit_delta_f64_workspace_bytes", n, G)
            work = torch.empty(nbytes, dtype=torch.uint8, device=dev)
            end = (P, G, lo, hi, refine, _ptr(ld), _ptr(idx), _ptr(work), nbytes, _stream(dev))
            if off:
                _lib.call("flmm_fit_delta_lowrank_f64", _ptr(s), n, _ptr(UY), n, _ptr(yy), n + off, *end)
            else:
                _lib.call("flmm_fit_delta_f64", _ptr(s), n, _ptr(UY), n, *end)
            got.append(ld)
    same = lambda x, y: bool(((x == y) | (torch.isnan(x) & torch.isnan(y))).all())
    assert same(got[0], got[2]) and same(got[1], got[3])


@pytest.mark.parametrize("C", [1, 4])
def test_gls_fit_by_warps(C):
    """Beyond ~12,000 samples a warp per column searches instead of two blocks."""
    from fasterlmm_gb300 import build, gls
    build()
    n, P = 12_900, 3
    s, Y, rn = _inputs(n, P, C)
    X = rn(C, n)
    ld, idx = gls.fit_delta_t(s, X, Y)

    def loss(x):
        sd = s[None, :] + x.exp()[:, None]
        w = 1.0 / sd
        L = torch.linalg.cholesky(torch.einsum("pn,cn,dn->pcd", w, X, X))
        z = torch.linalg.solve_triangular(L, torch.einsum("pn,cn,pn->pc", w, X, Y)[:, :, None], upper=False)[:, :, 0]
        rwr = (w * Y * Y).sum(1) - (z * z).sum(1)
        return n * (math.log(2 * math.pi) + torch.log(rwr / n) + 1.0) + torch.log(sd).sum(1)

    want, i = _golden(loss, P, s.device)
    assert torch.equal(idx.long(), i)
    torch.testing.assert_close(loss(ld), loss(want), rtol=4 * n * 2.0 ** -53, atol=1e-10)
