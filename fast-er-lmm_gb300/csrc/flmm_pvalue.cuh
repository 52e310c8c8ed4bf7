// -log10 of the F(1, df2) upper tail, the CLI's p-value (fasterlmm/cli.py:405-406, scipy.stats.f.sf(F, 1, df2)),
// computed in log space so that very large F gives a finite value instead of underflowing to p = 0.
//
// P(F(1, n) > F) = I_x(a, 1/2) with a = n / 2, x = n / (n + F), the regularized incomplete beta function, on the side of
// the symmetry I_x(a, b) = 1 - I_{1-x}(b, a) that converges fast:
//   * x < (a + 1) / (a + b + 2): the continued fraction for I_x(a, 1/2) (Abramowitz & Stegun 26.5.8);
//   * else, with y = 1 - x: I_y(1/2, a) = y^(1/2) x^a / (1/2 B(1/2, a)) sum_k (a + 1/2)_k / (3/2)_k y^k (A&S 26.5.4 and
//     15.1.1), positive terms.
// GB300's FP64 pipe runs at 1/60 of FP32 and a division costs a dozen of its operations, so neither loop divides: the
// coefficients of both depend on n alone and stand in a table, the fraction is the quotient of its forward
// recurrence's numerator and denominator (three operations a step), and convergence is tested by cross-multiplication.
// The prefactor takes sqrt(y) instead of a second logarithm.  One evaluation over 6.4 million statistics took 44 ms as
// Lentz's algorithm (four divisions a step); with the same error (that of lgamma in B).
#pragma once

#ifdef __CUDACC__
#define FLMM_HD __host__ __device__ __forceinline__
#else
#define FLMM_HD inline
#endif

#include <math.h>

namespace flmm {

// Constants of one df2, and tables of the first `n` coefficients (n = 0: formed where they are used).
struct FTail {
    double df2, a;          // a = df2 / 2
    double lbeta_a;         // log B(a, 1/2) + log a
    double two_over_beta;   // 2 / B(a, 1/2)
    double f_switch;        // F where x = (a + 1) / (a + 5/2): above it the fraction, below it the series
    const double* fraction; // [k - 1] for k = 1..n
    const double* series;   // [k] for k = 0..n - 1
    int n;
};

constexpr int kTailTable = 64;

// d_k / x of 1 / (1 + d_1 / (1 + d_2 / ...)) for I_x(a, 1/2)
FLMM_HD double tail_fraction_coef(double a, int k) {
    const double m = k / 2;
    if (k & 1) return -(a + m) * (a + 0.5 + m) / ((a + 2 * m) * (a + 2 * m + 1.0));
    return m * (0.5 - m) / ((a + 2 * m - 1.0) * (a + 2 * m));
}

FLMM_HD double tail_series_coef(double a, int k) { return (a + 0.5 + k) / (1.5 + k); }

FLMM_HD double tail_fraction(const FTail& t, double x) {
    double a0 = 0.0, a1 = 1.0, b0 = 1.0, b1 = 1.0;  // convergents k - 1 and k
    for (int k = 1; k <= 8000; k += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double d = (k + j <= t.n ? t.fraction[k + j - 1] : tail_fraction_coef(t.a, k + j)) * x;
            const double a2 = fma(d, a0, a1), b2 = fma(d, b0, b1);
            a0 = a1;
            a1 = a2;
            b0 = b1;
            b1 = b2;
        }
        if (fabs(fma(a1, b0, -a0 * b1)) <= 1e-16 * fabs(a1 * b1)) break;
        if (fabs(b1) < 0x1p-300) {  // both shrink together when a is large
            a0 *= 0x1p300;
            a1 *= 0x1p300;
            b0 *= 0x1p300;
            b1 *= 0x1p300;
        }
    }
    return a1 / b1;
}

FLMM_HD double tail_series(const FTail& t, double y) {
    double s = 1.0, term = 1.0;
    for (int k = 0; k < 4000; k += 2) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            term *= (k + j < t.n ? t.series[k + j] : tail_series_coef(t.a, k + j)) * y;
            s += term;
        }
        if (term < 1e-17 * s) break;
    }
    return s;
}

// P(F(1, df2) > F) for F > 0 and finite, returned as one of two terms: true with v = log p (the fraction for I_x(a, 1/2)
// itself), or false with v = I_y(1/2, a) = 1 - p.
FLMM_HD bool fsf_terms(double F, const FTail& t, double& v) {
    const double lx = -t.a * log1p(F / t.df2);  // a log x
    const double y = F / (t.df2 + F);           // 1 - x without cancellation
    if (F > t.f_switch) {
        v = lx + log(tail_fraction(t, t.df2 / (t.df2 + F)) * sqrt(y)) - t.lbeta_a;
        return true;
    }
    v = exp(lx) * sqrt(y) * t.two_over_beta * tail_series(t, y);
    return false;
}

// -log10 P(F(1, df2) > F).  F <= 0 gives 0 (p = 1); NaN propagates.
FLMM_HD double neglog10_fsf(double F, const FTail& t) {
    if (!(F > 0.0)) return (F == F) ? 0.0 : F;
    if (isinf(F)) return INFINITY;
    double v;
    const double logp = fsf_terms(F, t, v) ? v : log1p(-v);
    return -logp / 2.302585092994045684;
}

// P(F(1, df2) > F) itself (scipy.stats.f.sf(F, 1, df2)): F <= 0 gives 1, +inf gives 0, NaN propagates.
FLMM_HD double fsf(double F, const FTail& t) {
    if (!(F > 0.0)) return (F == F) ? 1.0 : F;
    if (isinf(F)) return 0.0;
    double v;
    return fsf_terms(F, t, v) ? exp(v) : 1.0 - v;
}

}  // namespace flmm
