"""
The F(1, df2) tail on either side of its switch between the continued fraction and the series, beyond the coefficient
tables, and the genomic inflation factor from the middle statistics, against scipy.

scipy and the library form log B(df2 / 2, 1 / 2) from lgamma values of size df2 log df2, whose rounding is the error left:
~df2 log(df2) 2^-53 relative to a tail exponent of order 1.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("df2", [1, 2, 3, 17, 994, 5000, 200_000])
def test_tail_matches_scipy(df2):
    from scipy.stats import f as fdist
    from fasterlmm_gb300 import build
    from fasterlmm_gb300.post import neg_log10_pvalue, pvalue
    build()
    rng = np.random.default_rng(df2)
    a = df2 / 2
    switch = df2 * ((a + 2.5) / (a + 1) - 1)  # F where x = (a + 1) / (a + 2.5)
    F = np.concatenate([rng.chisquare(1, 400), switch * (1 + rng.uniform(-1e-3, 1e-3, 100)), 10.0 ** rng.uniform(-14, 0, 50),
                        10.0 ** rng.uniform(0, 2.5, 200), [0.0, -1.0, np.inf, np.nan]])
    got = neg_log10_pvalue(torch.from_numpy(F).cuda(), df2).cpu().numpy()
    p = pvalue(torch.from_numpy(F).cuda(), df2).cpu().numpy()
    assert list(got[-4:-1]) == [0.0, 0.0, np.inf] and np.isnan(got[-1])
    assert list(p[-4:-1]) == [1.0, 1.0, 0.0] and np.isnan(p[-1])
    # (sf takes n / (n + F) near 1, which has lost F's digits where F is small; cdf takes F / (n + F))
    want = np.where(F[:-4] < 1.0, 1.0 - fdist.cdf(F[:-4], 1, df2), fdist.sf(F[:-4], 1, df2))
    ok = want > 1e-280
    tol = 1e-12 + 8 * df2 * np.log(df2 + 1.0) * 2.0 ** -53
    np.testing.assert_allclose(p[:-4][ok], want[ok], rtol=tol)
    # -log10 p near 0 carries the tail's absolute error
    np.testing.assert_allclose(got[:-4][ok], -np.log10(want[ok]), rtol=tol, atol=tol)


@pytest.mark.parametrize("M", [1, 2, 101, 1000])
def test_lambda_is_the_median_quantile(M):
    from scipy.stats import chi2, f as fdist
    from fasterlmm_gb300 import build
    from fasterlmm_gb300.post import lambda_gc
    build()
    rng = np.random.default_rng(M)
    F = rng.chisquare(1, (M, 4))
    F[rng.random((M, 4)) < 0.2] = np.nan
    F[:, 3] = np.nan
    F[0, 0] = np.inf
    lam, n = lambda_gc(torch.from_numpy(F).cuda(), 60)
    assert n.tolist() == (~np.isnan(F)).sum(0).tolist()
    for b in range(4):
        v = F[~np.isnan(F[:, b]), b]
        if v.size == 0:
            assert np.isnan(lam[b].item())
            continue
        want = np.median(chi2.isf(fdist.sf(v, 1, 60), 1)) / chi2.ppf(0.5, 1)
        np.testing.assert_allclose(lam[b].item(), want, rtol=1e-10)
