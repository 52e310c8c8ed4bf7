"""
The epistasis Wald's permutation columns, whose tests are ranked without forming every F, against the same columns as real ones,
whose F all come from the formula: the same largest F and the same first column, bit for bit, with tied, nearly tied,
near-self and strongly associated columns, on both sides of the setup's covariate counts and of its sample tiles.
"""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,C,M,P", [(60, 1, 40, 3), (255, 6, 700, 5), (257, 6, 300, 4), (300, 32, 513, 3), (300, 33, 257, 3)])
def test_ranked_maximum_is_the_formulas(N, C, M, P):
    from fasterlmm_gb300 import build, epi
    build()
    g = torch.Generator(device="cuda").manual_seed(N + C)
    rn = lambda *a: torch.randn(*a, generator=g, device="cuda", dtype=torch.float64)
    s, X, Y, ld, S = rn(N).abs() * 2, rn(1, N, C), rn(N, P), rn(P), rn(1, N, M)
    S[:, :, M // 2] = S[:, :, 3]                         # tied
    S[:, :, 11] = S[:, :, 9] * (1 + 1e-14)               # nearly tied
    S[:, :, 12] = -S[:, :, 9]
    S[:, :, 5] = 2 * X[:, :, 0]                          # in the span of the covariates
    Y[:, 1] = 3 * S[0, :, 9]                             # explained in full
    Y[:, 2] = S[0, :, 9] + 0.3 * Y[:, 2]
    *_, f_full, at_full = epi.snp_wald_scan_batched(s, X, Y, ld, S, n_real=P)
    *_, f_rank, at_rank = epi.snp_wald_scan_batched(s, X, Y, ld, S, n_real=1)
    assert torch.equal(f_full, f_rank) and torch.equal(at_full, at_rank)
