"""
Row kernels that work a block or a pass at a time: the dosage standardiser (few distinct values, or any), the covariate
regress-out at every specialised width and beyond, the low-rank variant operands, and the orthonormalisation of long
runs of equal eigenvalues.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dev():
    from fasterlmm_gb300 import build
    build()
    return torch.device("cuda", torch.cuda.current_device())


@pytest.mark.parametrize("N", [1, 31, 255, 256, 257, 1500])
@pytest.mark.parametrize("top", [2, 3, 127])
def test_dosage_standardiser(N, top):
    """Each value is (v - mean) / sd of exact integer sums, rounded as numpy rounds the same expressions."""
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    dev = _dev()
    rng = np.random.default_rng(N * 7 + top)
    G = rng.integers(-1, top + 1, size=(9, N)).astype(np.int8)
    G[1], G[2] = 1, -1          # no variance, no calls
    Gd = torch.from_numpy(G).to(dev)
    Z = torch.empty((9, N), dtype=torch.float64, device=dev)
    _lib.call("flmm_standardise_dosage", _ptr(Gd), N, N, 9, _ptr(Z), N, _stream(dev))
    for g, z in zip(G.astype(np.int64), Z.cpu().numpy()):
        ok = g >= 0
        n, s, q = max(int(ok.sum()), 1), int(g[ok].sum()), int((g[ok] ** 2).sum())
        sd = np.sqrt(np.float64(n * q - s * s)) / np.float64(n)
        with np.errstate(divide="ignore"):
            want = np.where(ok, (g - np.float64(s) / np.float64(n)) / (sd if sd else np.inf), 0.0)
        np.testing.assert_array_equal(z, want)


@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 6, 7, 8, 9, 64])
@pytest.mark.parametrize("rows,N", [(1, 70), (19, 333)])
def test_regress_out(D, rows, N):
    from fasterlmm_gb300.core import CovariateBasis
    dev = _dev()
    g = torch.Generator(device=dev).manual_seed(D)
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    X, A = rn(N, D), rn(rows, N)
    R = CovariateBasis(X).regress_out(A)
    want = A - (A @ torch.linalg.pinv(X).T) @ X.T
    # N-term and D-term sums of O(1) numbers
    torch.testing.assert_close(R, want, rtol=0, atol=64 * N * 2.0 ** -53)


@pytest.mark.parametrize("k,N", [(1, 1), (5, 33), (40, 511), (300, 513), (7, 11_000), (3, 56_321)])
def test_lowrank_variant_operands(k, N):
    """[US | S_r - C] and [US^2 | ||S_r - C||^2] as FP16 pairs: ~2^-21 of each row's largest entry; N = 56,321 is past the
    rows that fit in shared memory."""
    from fasterlmm_gb300 import _lib
    from fasterlmm_gb300.core import _ptr, _stream
    dev = _dev()
    g = torch.Generator(device=dev).manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float32)
    M = 3
    US, Ct, Sr = rn(M, k), rn(M, N), rn(M, N).double()
    ldb, ld2 = (k + N + 7) // 8 * 8, (k + 8) // 8 * 8
    h = lambda ld: torch.zeros(M, ld, dtype=torch.float16, device=dev)
    B1h, B1l, B2h, B2l = h(ldb), h(ldb), h(ld2), h(ld2)
    s1, s2 = (torch.empty(M, dtype=torch.float32, device=dev) for _ in range(2))
    _lib.call("flmm_lr_prep_variants", _ptr(US), k, _ptr(Sr), N, _ptr(Ct), N, M, k, N, None, N, 0, _ptr(B1h), _ptr(B1l),
              ldb, _ptr(s1), _ptr(B2h), _ptr(B2l), ld2, _ptr(s2), _stream(dev))
    res = Sr - Ct.double()
    want1 = torch.cat([US.double(), res], 1)
    want2 = torch.cat([US.double() ** 2, (res ** 2).sum(1, keepdim=True)], 1)
    for hi, lo, sc, want in ((B1h, B1l, s1, want1), (B2h, B2l, s2, want2)):
        got = (hi.double() + lo.double())[:, :want.shape[1]] * sc.double()[:, None]
        top = want.abs().max(1, keepdim=True).values
        assert float(((got - want).abs() / top).max()) < 2.0 ** -21


@pytest.mark.parametrize("N,run", [(64, 20), (200, 33), (300, 140)])
def test_long_runs_of_equal_eigenvalues(N, run):
    """The own FP32 solver on a Gram padded with a multiple of the identity, as the batched low-rank bases pad theirs:
    residual and orthogonality of an FP32 decomposition (a few 1e-7 of the norm, 50)."""
    from fasterlmm_gb300 import _lib, fast
    dev = _dev()
    g = torch.Generator(device=dev).manual_seed(N)
    G = torch.randn(N - run, 2 * N, generator=g, device=dev, dtype=torch.float64) / (2 * N) ** 0.5
    A = torch.zeros(1, N, N, device=dev, dtype=torch.float64)
    A[0, :N - run, :N - run] = G @ G.T
    d = torch.arange(N - run, N, device=dev)
    A[0, d, d] = -50.0
    U, ev = fast._eigh_batched_f32(_lib.context(dev.index), A)
    U, ev = U[0].double(), ev[0].double()
    assert float((U @ U.T - torch.eye(N, device=dev, dtype=torch.float64)).abs().max()) < 2e-5
    assert float((A[0] @ U.T - U.T * ev).abs().max()) < 50 * 2e-5
