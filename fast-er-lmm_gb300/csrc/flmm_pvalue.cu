// The F(1, df2) tail in FP64 over an array of F statistics, as p or -log10 p (the CLI's post-scan step,
// fasterlmm/cli.py:405-406); the maths is in flmm_pvalue.cuh.
#include <math.h>

#include "flmm_common.cuh"
#include "flmm_pvalue.cuh"

using namespace flmm;

namespace {

// The block's copy of `t` with its coefficient tables in shared memory.
__device__ __forceinline__ FTail with_tables(FTail t) {
    __shared__ double fraction[kTailTable], series[kTailTable];
    for (int k = threadIdx.x; k < kTailTable; k += blockDim.x) {
        fraction[k] = tail_fraction_coef(t.a, k + 1);
        series[k] = tail_series_coef(t.a, k);
    }
    __syncthreads();
    t.fraction = fraction;
    t.series = series;
    t.n = kTailTable;
    return t;
}

FTail tail_of(int df2) {
    const double a = 0.5 * df2;
    const double lbeta = lgamma(a) + lgamma(0.5) - lgamma(a + 0.5);
    return FTail{static_cast<double>(df2), a, lbeta + log(a), 2.0 * exp(-lbeta), 1.5 * df2 / (a + 1.0), nullptr, nullptr, 0};
}

enum class Tail { kNegLog10, kP, kChisq };

template <Tail WHAT>
__device__ __forceinline__ double tail_value(double F, const FTail& t) {
    if constexpr (WHAT == Tail::kNegLog10) return neglog10_fsf(F, t);
    const double p = fsf(F, t);
    if constexpr (WHAT == Tail::kP) return p;
    // 1-df chi-square quantile of the test's p-value, the input of the genomic inflation factor
    // (fasterlmm/inflation.py:19-29): chi2.isf(p, 1) = (Phi^-1(1 - p / 2))^2 = 2 erfcinv(p)^2.  NaN F gives NaN; p below
    // the FP64 range gives +inf, as scipy's isf(0).
    const double z = erfcinv(p);
    return isnan(p) ? NAN : 2.0 * z * z;
}

// out[i] = the tail of F[i].  Under the null one statistic in twelve lies past the switch to the continued fraction, so
// nearly every warp would run both forms one after the other (6.4 million: 13 ms against 4): a block sorts
// kTailChunk statistics by form into two lists first and runs each list densely.
constexpr int kTailThreads = 256, kTailChunk = 2048;

template <Tail WHAT>
__global__ void __launch_bounds__(kTailThreads)
k_tail(const double* __restrict__ F, int64_t n, FTail tail, double* __restrict__ out) {
    const FTail t = with_tables(tail);
    __shared__ uint16_t list[kTailChunk];  // series forms from the front, fractions from the back
    __shared__ int count[2];
    const unsigned lane = threadIdx.x & 31;
    for (int64_t i0 = blockIdx.x * static_cast<int64_t>(kTailChunk); i0 < n;
         i0 += static_cast<int64_t>(gridDim.x) * kTailChunk) {
        const int m = static_cast<int>(n - i0 < kTailChunk ? n - i0 : kTailChunk);
        if (threadIdx.x < 2) count[threadIdx.x] = 0;
        __syncthreads();
        for (int k0 = 0; k0 < m; k0 += kTailThreads) {
            const int k = k0 + threadIdx.x;
            const bool in = k < m, frac = in && F[i0 + k] > t.f_switch;
            const unsigned all = __ballot_sync(0xffffffffu, in), fr = __ballot_sync(0xffffffffu, frac);
            int at_s = 0, at_f = 0;
            if (lane == 0) {
                at_s = atomicAdd(count, __popc(all & ~fr));
                at_f = atomicAdd(count + 1, __popc(fr));
            }
            at_s = __shfl_sync(0xffffffffu, at_s, 0);
            at_f = __shfl_sync(0xffffffffu, at_f, 0);
            const unsigned below = (1u << lane) - 1u;
            const int place = frac ? m - 1 - (at_f + __popc(fr & below)) : at_s + __popc(all & ~fr & below);
            if (in) list[place] = static_cast<uint16_t>(k);
        }
        __syncthreads();
        // the lists start on warp boundaries of their own, so no warp holds both
        const int ns = count[0], ns_pad = (ns + 31) & ~31, total = ns_pad + count[1];
        for (int q = threadIdx.x; q < total; q += kTailThreads) {
            if (q >= ns && q < ns_pad) continue;
            const int k = list[q < ns ? q : q - ns_pad + ns];
            out[i0 + k] = tail_value<WHAT>(F[i0 + k], t);
        }
        __syncthreads();
    }
}

template <Tail WHAT>
int launch_tail(const double* F, int64_t n, int df2, double* out, cudaStream_t st) {
    int sms = 0;
    const int rc = sm_count(&sms);
    if (rc) return rc;
    const int64_t chunks = (n + kTailChunk - 1) / kTailChunk, most = 8 * static_cast<int64_t>(sms);
    k_tail<WHAT><<<static_cast<unsigned>(chunks < most ? chunks : most), kTailThreads, 0, st>>>(F, n, tail_of(df2), out);
    return check_launch("k_tail");
}

// Genome-wide threshold per phenotype (fasterlmm/cli.py:128): p = P(F(1, df2) > perm_max_F) for the row's n_perm
// permutation maxima, then numpy.quantile(p, q) with linear interpolation between order statistics.  p is
// decreasing in F, so the ascending p order is the descending F order: the row is sorted once (bitonic, shared
// memory) and only the two straddling order statistics are converted to p.  One block per phenotype.
__global__ void k_perm_threshold(const double* __restrict__ pmax, int B, int n_perm, int npow2, FTail tail,
                                 double q, double* __restrict__ thresh) {
    extern __shared__ double v[];
    const int b = blockIdx.x;
    const double* row = pmax + static_cast<int64_t>(b) * n_perm;
    for (int i = threadIdx.x; i < npow2; i += blockDim.x) v[i] = (i < n_perm) ? -row[i] : INFINITY;  // -F ascending
    __syncthreads();
    for (int size = 2; size <= npow2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < npow2 / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1));
                const int hi = lo + stride;
                const bool up = (lo & size) == 0;
                const double a = v[lo], c = v[hi];
                if ((a > c) == up) {
                    v[lo] = c;
                    v[hi] = a;
                }
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        // numpy's default ("linear"): position h = (n - 1) q, value = x[floor h] + (h - floor h)(x[floor h + 1] - x[floor h])
        const double h = (n_perm - 1) * q;
        const int j = static_cast<int>(floor(h));
        const double frac = h - j;
        const double p0 = fsf(-v[j], tail);
        double out = p0;
        if (frac > 0.0 && j + 1 < n_perm) {
            const double p1 = fsf(-v[j + 1], tail);
            out = p0 + frac * (p1 - p0);
        }
        thresh[b] = out;
    }
}

}  // namespace

extern "C" int flmm_perm_threshold_p(const double* perm_max_F, int B, int n_perm, int df2, double q, double* thresh,
                                     void* stream) {
    FLMM_REQUIRE((perm_max_F && thresh) || B == 0, "flmm_perm_threshold_p: NULL argument");
    FLMM_REQUIRE(n_perm >= 1 && n_perm <= 16384 && df2 >= 1 && q >= 0.0 && q <= 1.0,
                 "flmm_perm_threshold_p: need 1 <= n_perm <= 16384, df2 >= 1, 0 <= q <= 1");
    if (B == 0) return FLMM_OK;
    int npow2 = 1;
    while (npow2 < n_perm) npow2 <<= 1;
    const size_t smem = sizeof(double) * npow2;
    // (one bound whatever n_perm: another host thread's call must not lower it under this launch)
    FLMM_CUDA(cudaFuncSetAttribute(k_perm_threshold, cudaFuncAttributeMaxDynamicSharedMemorySize, 16384 * sizeof(double)));
    k_perm_threshold<<<B, 256, smem, as_stream(stream)>>>(perm_max_F, B, n_perm, npow2, tail_of(df2), q, thresh);
    return check_launch("k_perm_threshold");
}

extern "C" int flmm_neglog10_pvalue(const double* F, int64_t n, int df2, double* out, void* stream) {
    FLMM_REQUIRE((F && out) || n == 0, "flmm_neglog10_pvalue: NULL argument");
    FLMM_REQUIRE(df2 >= 1, "flmm_neglog10_pvalue: df2 must be >= 1 (got %d)", df2);
    if (n == 0) return FLMM_OK;
    return launch_tail<Tail::kNegLog10>(F, n, df2, out, as_stream(stream));
}

extern "C" int flmm_chisq1_from_f(const double* F, int64_t n, int df2, double* out, void* stream) {
    FLMM_REQUIRE((F && out) || n == 0, "flmm_chisq1_from_f: NULL argument");
    FLMM_REQUIRE(df2 >= 1, "flmm_chisq1_from_f: df2 must be >= 1 (got %d)", df2);
    if (n == 0) return FLMM_OK;
    return launch_tail<Tail::kChisq>(F, n, df2, out, as_stream(stream));
}

extern "C" int flmm_f_pvalue(const double* F, int64_t n, int df2, double* out, void* stream) {
    FLMM_REQUIRE((F && out) || n == 0, "flmm_f_pvalue: NULL argument");
    FLMM_REQUIRE(df2 >= 1, "flmm_f_pvalue: df2 must be >= 1 (got %d)", df2);
    if (n == 0) return FLMM_OK;
    return launch_tail<Tail::kP>(F, n, df2, out, as_stream(stream));
}
