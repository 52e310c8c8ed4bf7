"""
The native chromosome loop of the fast form against the same loop run from Python (which a progress callback selects): the
same bits, for LOCO and single-kinship scans, unsorted labels, a separate kinship panel that lacks a chromosome, chromosomes
of one variant, one stream or two, and with the strong-test re-evaluation on or off.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scan(monkeypatch, python: bool, **kw):
    from fasterlmm_gb300 import build, fast
    build()
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(kw.pop("seed", 1))
    rn = lambda *s: torch.randn(*s, generator=g, device=dev, dtype=torch.float64)
    N, M, D, P, B = kw.pop("shape")
    std = lambda Z: (Z - Z.mean(1, keepdim=True)) / Z.std(1, unbiased=False, keepdim=True)
    Zt = std(rn(M, N))
    X = torch.cat([torch.ones(N, 1, device=dev, dtype=torch.float64), rn(N, D - 1)], 1)
    Yt = rn(P, N)
    Yt[0] += 3.0 * Zt[M // 2]  # a strong association
    kin = kw.pop("kin", None)
    if kin is not None:
        kw.update(Zt_kin=std(rn(kin.size, N)), chrom_kin=kin)
    for k, v in kw.pop("patch", {}).items():
        monkeypatch.setattr(fast, k, v)
    calls = []
    res = fast.scan_t(Zt, X, Yt, kw.pop("chrom"), n_real=B, on_chrom=(lambda *a: calls.append(a)) if python else None, **kw)
    return res, calls


@pytest.mark.parametrize("case", [
    dict(shape=(40, 30, 1, 5, 2), chrom=np.repeat([1, 2, 3], 10)),
    dict(shape=(131, 257, 3, 70, 70), chrom=np.tile([5, 2, 9], 86)[:257]),
    dict(shape=(90, 64, 2, 33, 4), chrom=np.r_[np.zeros(1), np.ones(62), [7]].astype(int)),
    dict(shape=(75, 120, 4, 9, 3), chrom=np.repeat([1, 2], 60), loco=False),
    dict(shape=(75, 120, 4, 9, 3), chrom=np.repeat([1, 2, 4], 40), kin=np.repeat([1, 2, 3], 50)),
    dict(shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), patch=dict(PIPELINE=False)),
    dict(shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), patch=dict(REFINE_F=None), n_grid=17, refine=False),
    dict(shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), patch=dict(REFINE_F=0.5, REFINE_CAP=8)),
    dict(shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), patch=dict(REFINE_CAP=1 << 40)),
    dict(shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), log_delta_min=0.5, log_delta_max=0.5),
    dict(shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), log_delta_min=0.5, log_delta_max=0.5, n_grid=1),
])
def test_native_loop_gives_the_python_loops_bits(monkeypatch, case):
    a, none = _scan(monkeypatch, False, **{**case})
    b, calls = _scan(monkeypatch, True, **{**case})
    n = len(b.log_delta)
    assert not none and calls == [(k + 1, n) for k in range(n)]
    for k in ("f", "beta", "se", "sfve", "nullh2", "max_F"):
        assert torch.equal(getattr(a, k), getattr(b, k)), k
    assert list(a.log_delta) == list(b.log_delta)
    assert all(torch.equal(a.log_delta[c], b.log_delta[c]) for c in a.log_delta)


@pytest.mark.parametrize("choice", [(2, 0, 1), (2, 1, 3)])
@pytest.mark.parametrize("shape,sizes", [((40, 30, 1, 5, 2), [1, 28, 1]), ((300, 700, 3, 270, 130), [129, 256, 0, 315]),
                                         ((129, 301, 1, 257, 257), [128, 127, 46])])
def test_units_together_and_one_by_one_give_the_same_bits(monkeypatch, shape, sizes, choice):
    """Every unit in one launch (CTA pairs) and unit by unit (single-CTA products forced), at the edges of a unit's tiles."""
    from fasterlmm_gb300 import _lib, build
    build()
    kw = dict(shape=shape, chrom=np.repeat(np.arange(len(sizes)), sizes), patch=dict(REFINE_F=1.0))
    a, _ = _scan(monkeypatch, False, **{**kw})
    try:
        _lib.tc_config(*choice)
        b, _ = _scan(monkeypatch, False, **{**kw})
        c, _ = _scan(monkeypatch, True, **{**kw})
    finally:
        _lib.tc_config(1)
    for k in ("f", "beta", "se", "sfve", "nullh2", "max_F"):
        assert torch.equal(getattr(a, k), getattr(b, k)) and torch.equal(getattr(a, k), getattr(c, k)), k


def test_a_chromosome_that_holds_every_variant_is_refused(monkeypatch):
    from fasterlmm_gb300 import _lib
    with pytest.raises(_lib.FlmmError):
        _scan(monkeypatch, False, shape=(40, 30, 1, 5, 2), chrom=np.zeros(30, dtype=int))


@pytest.mark.parametrize("python", [False, True])
def test_one_sample_more_than_covariates_is_refused(monkeypatch, python):
    """F would have no degrees of freedom."""
    from fasterlmm_gb300 import _lib
    with pytest.raises(_lib.FlmmError):
        _scan(monkeypatch, python, shape=(9, 60, 8, 20, 3), chrom=np.repeat([1, 2, 3], 20))


@pytest.mark.parametrize("kw", [dict(log_delta_min=float("nan")), dict(log_delta_max=float("inf")),
                                dict(log_delta_min=2.0, log_delta_max=-2.0)])
def test_bad_delta_ranges_are_refused(monkeypatch, kw):
    from fasterlmm_gb300 import _lib
    with pytest.raises((_lib.FlmmError, ValueError, OverflowError)):
        _scan(monkeypatch, False, shape=(60, 80, 2, 40, 6), chrom=np.repeat([1, 2], 40), **kw)
