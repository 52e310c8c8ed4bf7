"""
GPU parity of the low-rank path (fasterlmm/lowrank.py) and its block engine (fasterlmm/extreme_scan.py) against the
reference's own outputs (tests/golden/lowrank_*.npz) at the reference's parity tolerance.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

import flmm_oracle as orc
from conftest import z_float
from parity import DETAIL, assert_scan_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module", autouse=True)
def _built():
    from fasterlmm_gb300 import build
    build()


def _np(res) -> dict:
    return {k: getattr(res, k).detach().cpu().double().numpy() for k in DETAIL + ("max_F",)}


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def test_lowrank_components_match_golden(golden):
    from fasterlmm_gb300 import lowrank
    g = golden("lowrank_components")
    for tag in ("lo", "hi"):
        spec = lowrank.lowrank_rotate(_t(g[f"{tag}_G"]), _t(g["X"]), _t(g["Y"]))
        assert spec.Neff == int(g[f"{tag}_Neff"])
        s = spec.s.cpu().numpy()
        big, gbig = s > 1e-12, g[f"{tag}_s"] > 1e-12   # see test_oracle_lowrank_components on the noise directions
        np.testing.assert_allclose(s[big], g[f"{tag}_s"][gbig], rtol=1e-7, atol=1e-10)
        np.testing.assert_allclose(spec.UY.cpu().numpy()[big] ** 2, g[f"{tag}_UY"][gbig] ** 2, rtol=1e-6, atol=1e-10)
        ld_grid = lowrank.fit_delta_grid_lowrank(spec, refine=False).cpu().numpy()
        assert np.array_equal(ld_grid, g[f"{tag}_log_delta_grid"])
        ld = lowrank.fit_delta_grid_lowrank(spec).cpu().numpy()
        assert np.abs(ld - g[f"{tag}_log_delta"]).max() < 1e-3
        res = lowrank.snp_wald_scan_lowrank(spec, torch.from_numpy(g[f"{tag}_log_delta"]), _t(g["S"]), n_real=2)
        got = _np(res)
        for k in DETAIL + ("max_F",):
            np.testing.assert_allclose(got[k], g[f"{tag}_{k}"], rtol=1e-7, atol=1e-10, err_msg=k)


def test_lowrank_loco_single_k_and_block_engines_match_golden(golden):
    from fasterlmm_gb300 import lowrank
    g = golden("lowrank_loco")
    Zs = orc.standardise_columns(z_float(g["G"]))
    Gs = orc.standardise_columns(z_float(g["G_kin"]))
    B = int(g["n_real"])
    seen = []
    res = lowrank.loco_scan_lowrank(_t(Gs), g["chrom_kin"], _t(Zs), g["chrom"], _t(g["X"]), _t(g["Y_all"]), n_real=B,
                                    on_chrom=lambda k, n: seen.append(k))
    assert seen == list(range(1, len(np.unique(g["chrom"])) + 1))
    assert_scan_close(_np(res), g)
    res1 = lowrank.single_k_scan_lowrank(_t(Gs), _t(Zs), _t(g["X"]), _t(g["Y_all"]), n_real=B)
    assert_scan_close(_np(res1), g, prefix="sk_")
    # resident blocks (host Z, blocks of 37 splitting chromosomes), FP64 and the FP32 default
    Zh = torch.from_numpy(Zs)
    r64 = lowrank.loco_scan_resident(Zh, g["chrom"], _t(Gs), g["chrom_kin"], _t(g["X"]), _t(g["Y_all"]), n_real=B,
                                     block_size=37, dtype=torch.float64)
    assert r64.f.device.type == "cpu" and r64.f.dtype == torch.float64
    assert_scan_close(_np(r64), g, prefix="res64_")
    r32 = lowrank.loco_scan_resident(Zh.float(), g["chrom"], _t(Gs), g["chrom_kin"], _t(g["X"]), _t(g["Y_all"]),
                                     n_real=B, block_size=37)
    assert r32.f.dtype == torch.float32
    # The FP32 default here is FP64 arithmetic rounded to FP32: it matches the reference's FP64 scan to FP32 rounding.
    # (The reference's own FP32 run, kept in the fixture as res32_*, is no oracle: its FP32 delta fit moves nullh2 by
    # up to 80 % and F by up to 40 % relative on flat-likelihood columns against its FP64 scan.)
    assert_scan_close(_np(r32), g, prefix="res64_", rtol=1e-6, atol_scale=1.0)
    # a streamed reader: host blocks produced on demand
    chrom = np.asarray(g["chrom"])

    def source(c):
        idx = np.flatnonzero(chrom == c)
        for b0 in range(0, idx.size, 50):
            cols = idx[b0:b0 + 50]
            yield Zs[:, cols], cols

    rs = lowrank.loco_scan_blocks(source, sorted(np.unique(chrom).tolist()), Zs.shape[1], _t(Gs), g["chrom_kin"],
                                  _t(g["X"]), _t(g["Y_all"]), n_real=B, dtype=torch.float64)
    assert_scan_close(_np(rs), g)


@pytest.mark.parametrize("sizes,N", [((20, 25, 30, 15), 200), ((30, 31), 100), ((300, 14, 26), 90), ((60, 14, 26), 90),
                                     ((700, 5), 64)])
def test_loco_bases_form_no_gram_larger_than_their_selections_need(monkeypatch, sizes, N):
    """The basis of every selection has basis_t's bits, whether its Gram is its own or a part of one for all rows, and no
    Gram has over twice the entries of the largest that a basis is taken from."""
    from fasterlmm_gb300 import lowrank
    g = torch.Generator(device=DEV).manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)
    chrom = torch.from_numpy(np.repeat(np.arange(len(sizes)), sizes)).to(DEV)
    Gt = rn(chrom.numel(), N)
    basis = lowrank.CovariateBasis(torch.cat([torch.ones(N, 1, device=DEV, dtype=torch.float64), rn(N, 2)], 1))
    keeps = [torch.nonzero(chrom != c).flatten() for c in range(len(sizes))]
    alone = [lowrank.basis_t(Gt[k], basis) for k in keeps]
    formed, rotate = [0], lowrank.rotate_rows
    monkeypatch.setattr(lowrank, "rotate_rows",
                        lambda A, B: (formed.append(A.shape[0] ** 2 if A is B else 0), rotate(A, B))[1])
    got = list(lowrank.loco_bases(Gt, keeps, basis))
    assert max(formed) <= 2 * max(min(k.numel(), N) for k in keeps) ** 2
    for (s, U), (s1, U1) in zip(got, alone, strict=True):
        assert torch.equal(s, s1) and torch.equal(U, U1)
