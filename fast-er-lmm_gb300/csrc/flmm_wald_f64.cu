// Plain FP64 form of the compat Wald scan (fasterlmm/core.py:601-671): the two per-chromosome products
// sWy = (w o UY)^T US and sWs = w^T (US o US), then beta, var_beta, F, SE, SFVE and the per-column genome max.
// The products are FP64 sums of Neff terms per test and bound by the FP64 pipe (1.08 TFLOP/s measured of ~1.25), so
// where they are large they run on the tensor cores from exact digit planes (flmm_oz64.cu) in blocks of columns and
// variants whose sums an epilogue kernel reads back (16 bytes per test); 1,100 columns x 4,096 variants x 995 with its
// rotation: 23.9 -> 1.32 ms.  Small products stay in the fused FP64 tile kernel, which needs one launch.
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "flmm_common.cuh"
#include "flmm_oz64.cuh"

using namespace flmm;

namespace {

// W[p, n] = 1 / (s[n] + exp(ld[p])), A1 = W o UY, rWr[p] = max(sum_n (W UY) UY, floor)
// (fasterlmm/core.py:639-643); one warp per column
__global__ void k_wald_prep(const double* __restrict__ s, int Neff, const double* __restrict__ UYt, int64_t ldu,
                            const double* __restrict__ ld, int P, double* __restrict__ W, double* __restrict__ A1,
                            double* __restrict__ rWr) {
    const int lane = threadIdx.x & 31;
    const int64_t p = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
    if (p >= P) return;
    const double delta = exp(ld[p]);
    const double* u = UYt + p * ldu;
    double acc = 0.0;
    for (int n = lane; n < Neff; n += 32) {
        double w = 1.0 / (s[n] + delta);
        double a = mul_rn(w, u[n]);
        W[p * Neff + n] = w;
        A1[p * Neff + n] = a;
        acc += mul_rn(a, u[n]);
    }
    acc = warp_sum(acc);
    if (lane == 0) rWr[p] = fmax(acc, kPosFloor);
}

constexpr int TP = 64, TM = 64, TK = 16, NT = 256;

// Thread (tx, ty) owns columns p0 + tx + 16 r and variants m0 + ty + 16 c, so the detail stores of consecutive tx
// (consecutive columns of one output row) coalesce.
__global__ void __launch_bounds__(NT)
k_wald_f64(const double* __restrict__ W, const double* __restrict__ A1, const double* __restrict__ rWr, int Neff,
           double var_df, int P, int n_real, const double* __restrict__ USt, int64_t ldus, int Mc,
           const int64_t* __restrict__ rows, double* __restrict__ f, double* __restrict__ beta, double* __restrict__ se,
           double* __restrict__ sfve, int64_t ldo, double* __restrict__ max_F) {
    __shared__ double Ws[TK][TP + 1];
    __shared__ double As[TK][TP + 1];
    __shared__ double Us[TK][TM + 1];
    __shared__ double U2s[TK][TM + 1];
    __shared__ double red[16][TP];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int p0 = blockIdx.y * TP, m0 = blockIdx.x * TM;
    double sy[4][4] = {}, ss[4][4] = {};
    for (int k0 = 0; k0 < Neff; k0 += TK) {
#pragma unroll
        for (int l = 0; l < (TP * TK) / NT; ++l) {
            int t = tid + l * NT, p = t / TK, k = t % TK;
            int gp = p0 + p, gk = k0 + k;
            bool ok = gp < P && gk < Neff;
            Ws[k][p] = ok ? W[static_cast<int64_t>(gp) * Neff + gk] : 0.0;
            As[k][p] = ok ? A1[static_cast<int64_t>(gp) * Neff + gk] : 0.0;
        }
#pragma unroll
        for (int l = 0; l < (TM * TK) / NT; ++l) {
            int t = tid + l * NT, m = t / TK, k = t % TK;
            int gm = m0 + m, gk = k0 + k;
            double v = (gm < Mc && gk < Neff) ? USt[static_cast<int64_t>(gm) * ldus + gk] : 0.0;
            Us[k][m] = v;
            U2s[k][m] = mul_rn(v, v);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            double a[4], w[4], u[4], u2[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) { a[r] = As[k][tx + 16 * r]; w[r] = Ws[k][tx + 16 * r]; }
#pragma unroll
            for (int c = 0; c < 4; ++c) { u[c] = Us[k][ty + 16 * c]; u2[c] = U2s[k][ty + 16 * c]; }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    sy[r][c] = fma(a[r], u[c], sy[r][c]);
                    ss[r][c] = fma(w[r], u2[c], ss[r][c]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int p = p0 + tx + 16 * r;
        const bool p_ok = p < P;
        const double rwr = p_ok ? rWr[p] : 1.0;
        double colmax = -INFINITY;
        bool col_nan = false;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int m = m0 + ty + 16 * c;
            if (!p_ok || m >= Mc) continue;
            // fasterlmm/core.py:651-655, in the reference's operation order
            const double swy = sy[r][c];
            const double denom = fmax(ss[r][c], kPosFloor);
            const double b = swy / denom;
            const double q = mul_rn(swy, swy);
            const double rss = fmax(add_rn(rwr, -(q / denom)), kPosFloor);
            const double var_b = (rss / var_df) / denom;
            const double F = mul_rn(b, b) / var_b;
            colmax = fmax(colmax, F);
            col_nan |= isnan(F);
            if (p < n_real) {
                const int64_t o = rows[m] * ldo + p;
                f[o] = F;
                beta[o] = b;
                se[o] = sqrt(var_b);
                sfve[o] = sqrt(fmax(q / mul_rn(denom, rwr), 0.0));
            }
        }
        red[ty][tx + 16 * r] = col_nan ? NAN : colmax;
    }
    __syncthreads();
    if (tid < TP && p0 + tid < P) {
        double v = -INFINITY;
        bool any_nan = false;
        for (int r = 0; r < 16; ++r) {
            double x = red[r][tid];
            any_nan |= isnan(x);
            v = fmax(v, x);
        }
        if (any_nan) v = NAN;
        if (v >= 0.0 || isnan(v)) atomic_max_nonneg(max_F + p0 + tid, v);
    }
}

// beta, F, SE and SFVE of one test from its two sums (fasterlmm/core.py:651-655, in the reference's operation order)
struct Test {
    double F, b, var_b, q, denom;
};

__device__ __forceinline__ Test wald_test(double swy, double sws, double rwr, double var_df) {
    Test t;
    t.denom = fmax(sws, kPosFloor);
    t.b = swy / t.denom;
    t.q = mul_rn(swy, swy);
    const double rss = fmax(add_rn(rwr, -(t.q / t.denom)), kPosFloor);
    t.var_b = (rss / var_df) / t.denom;
    t.F = mul_rn(t.b, t.b) / t.var_b;
    return t;
}

// Epilogue over the sums of a block of columns and variants (layout: flmm_oz64.cuh): a thread block takes 32 columns x
// kFinTile variants, transposed through shared memory so that the reads run along the variants and the detail stores along
// the columns.  Real columns get the full epilogue; with 256 variants a block, those few blocks' FP64 pipes set the time
// (1,100 columns, 100 of them real, x 4,096: 265 -> 161 us with one F a block; 660 with covariates, 60 real, x 4,000:
// 277 -> 138).  A permutation column needs its
// largest F only, and F grows with q / denom, so its tests are ranked by cross-multiplication (three FP64 operations
// instead of four divisions; GB300's FP64 pipe is the bound here) and one F is formed per block; sums outside
// 1e-100 .. 1e100, and NaN, take the full formula.
constexpr int kFinP = 32, kFinTile = 64;

template <bool GLS>
__global__ void __launch_bounds__(256)
k_wald_finish(const double* __restrict__ Gy, const double* __restrict__ Gs, const double* __restrict__ Gq, int nq,
              int64_t ldg, const double* __restrict__ rWr, double var_df, int P, int n_real, int Mc,
              const int64_t* __restrict__ rows, double* __restrict__ f, double* __restrict__ beta,
              double* __restrict__ se, double* __restrict__ sfve, int64_t ldo, double* __restrict__ max_F) {
    __shared__ double sy[kFinP][kFinTile + 1];
    __shared__ double ss[kFinP][kFinTile + 1];
    __shared__ double red[8][kFinP], red_q[8][kFinP], red_den[8][kFinP], red_sy[8][kFinP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p0 = blockIdx.y * kFinP, p = p0 + lane;
    const bool p_ok = p < P, real = p < n_real;
    const double rwr = p_ok ? rWr[p] : 1.0;
    double best = -INFINITY, bq = -1.0, bden = 1.0, bsy = 0.0;
    bool any_nan = false;
    const int m0 = blockIdx.x * kFinTile, m_end = min(Mc, m0 + kFinTile);
#pragma unroll
    for (int l = 0; l < kFinP * kFinTile / 256; ++l) {
        const int t = tid + l * 256, r = t / kFinTile, c = t % kFinTile;
        if (p0 + r < P && m0 + c < m_end) {
            const int64_t o = static_cast<int64_t>(p0 + r) * ldg + m0 + c;
            sy[r][c] = Gy[o];
            double w = Gs[o];
            if (GLS) {
                const double* g = Gq + static_cast<int64_t>(p0 + r) * nq * ldg + m0 + c;
                double quad = 0.0;
                for (int k = 0; k < nq; ++k) quad = fma(g[k * ldg], g[k * ldg], quad);
                w = add_rn(w, -quad);
            }
            ss[r][c] = w;
        }
    }
    __syncthreads();
    for (int c = warp; p_ok && c < kFinTile && m0 + c < m_end; c += 8) {
        const double swy = sy[lane][c], den = fmax(ss[lane][c], kPosFloor), q = mul_rn(swy, swy);
        if (!real && q < 1e100 && den < 1e100 && den > 1e-100) {
            if (q * bden > bq * den) {
                bq = q;
                bden = den;
                bsy = swy;
            }
            continue;
        }
        const Test t = wald_test(swy, ss[lane][c], rwr, var_df);
        best = fmax(best, t.F);
        any_nan |= isnan(t.F);
        if (real) {
            const int64_t o = rows[m0 + c] * ldo + p;
            f[o] = t.F;
            beta[o] = t.b;
            se[o] = sqrt(t.var_b);
            sfve[o] = sqrt(fmax(t.q / mul_rn(t.denom, rwr), 0.0));
        }
    }
    red[warp][lane] = any_nan ? NAN : best;
    red_q[warp][lane] = bq;
    red_den[warp][lane] = bden;
    red_sy[warp][lane] = bsy;
    __syncthreads();
    if (warp == 0 && p_ok) {
        double v = -INFINITY;
        bool nan = false;
        for (int r = 0; r < 8; ++r) {
            nan |= isnan(red[r][lane]);
            v = fmax(v, red[r][lane]);
        }
        // one F a column for its best ranked test
        for (int r = 1; r < 8; ++r) {
            const double q = red_q[r][lane], den = red_den[r][lane];
            if (q * bden > bq * den) {
                bq = q;
                bden = den;
                bsy = red_sy[r][lane];
            }
        }
        if (bq >= 0.0) {
            const double F = wald_test(bsy, bden, rwr, var_df).F;
            v = fmax(v, F);
            nan |= isnan(F);
        }
        if (nan) v = NAN;
        if (v >= 0.0 || isnan(v)) atomic_max_nonneg(max_F + p, v);
    }
}

// The scan runs over blocks of at most kBlockP columns x kBlockM variants, fewer where their digit planes (32 bytes
// per element of a column or variant) would pass kPlaneBytes: the workspace does not grow with P or Mc.  A shorter workspace
// gets smaller blocks, and the FP64 tile kernel's, which has no planes or sums in memory, where the smallest do not fit.
constexpr int kBlockP = 2048, kBlockM = 4096;
constexpr size_t kPlaneBytes = size_t(256) << 20;

int block_rows(int most, int unit, int K) {
    const size_t fit = kPlaneBytes / (32 * static_cast<size_t>(K)) / unit * unit;
    return static_cast<int>(fit < static_cast<size_t>(unit) ? unit : fit < static_cast<size_t>(most) ? fit : most);
}

struct WaldWs {
    bool tensor;
    int pc, mc;                // columns and variants of a block
    double *rWr, *A1, *W, *G;  // A1 and W adjacent (pc, Neff) matrices; G (2, pc, mc)
    char *cols, *vars;         // digit operands of [A1 | W] and [US | US^2]
    int* bal;                  // balancing exponents and their scratch
    size_t bytes;
};

// Columns of the FP64 tile kernel that `bytes` hold; all of P in the shortest workspace that is taken.
size_t tile_bytes(int P, int Neff) { return sizeof(double) * static_cast<size_t>(P) * (2 * static_cast<size_t>(Neff) + 1) + 512; }

WaldWs carve_blocks(void* base, int pc, int mc, int Neff) {
    WaldWs w{};
    w.tensor = true;
    w.pc = pc;
    w.mc = mc;
    size_t off = 0;
    const uintptr_t b = reinterpret_cast<uintptr_t>(base);
    const uintptr_t b0 = (b + 1023) / 1024 * 1024;
    auto take = [&](size_t n) {
        const uintptr_t p = b0 + off;
        off += (n + 1023) / 1024 * 1024;
        return p;
    };
    w.rWr = reinterpret_cast<double*>(take(sizeof(double) * w.pc));
    w.A1 = reinterpret_cast<double*>(take(2 * sizeof(double) * static_cast<size_t>(w.pc) * Neff));
    w.W = w.A1 + static_cast<size_t>(w.pc) * Neff;
    w.G = reinterpret_cast<double*>(take(2 * sizeof(double) * static_cast<size_t>(w.pc) * w.mc));
    w.cols = reinterpret_cast<char*>(take(oz_operand_bytes(w.pc, Neff, 2, kOzRowsA)));
    w.vars = reinterpret_cast<char*>(take(oz_operand_bytes(w.mc, Neff, 2, kOzRowsB)));
    w.bal = reinterpret_cast<int*>(take(sizeof(int) * oz_balance_ints(Neff)));
    w.bytes = off + 1024;
    return w;
}

// The blocks of a scan of P columns x Mc variants in `bytes` of workspace.
WaldWs carve_wald(void* base, int P, int Neff, int Mc, size_t bytes) {
    int pc = block_rows(kBlockP, kOzRowsA, Neff), mc = block_rows(kBlockM, kOzRowsB, Neff);
    if (P < pc) pc = P > 0 ? P : 1;
    const int most = (Mc > 0 ? (Mc - 1) / kOzRowsB + 1 : 1) * kOzRowsB;
    if (most < mc) mc = most;
    for (; oz_worth(pc, Mc < mc ? Mc : mc, Neff);) {
        const WaldWs w = carve_blocks(base, pc, mc, Neff);
        if (w.bytes <= bytes) return w;
        if (mc > 512 || (pc <= kOzRowsA && mc > kOzRowsB)) mc = (mc / 2 + kOzRowsB - 1) / kOzRowsB * kOzRowsB;
        else if (pc > kOzRowsA) pc = (pc / 2 + kOzRowsA - 1) / kOzRowsA * kOzRowsA;
        else break;
    }
    WaldWs w{};
    w.mc = Mc;
    w.A1 = static_cast<double*>(base);
    const size_t column = sizeof(double) * (2 * static_cast<size_t>(Neff) + 1);
    const size_t fit = bytes / column;
    w.pc = fit < static_cast<size_t>(P) ? static_cast<int>(fit) : P;
    w.W = w.A1 + static_cast<size_t>(w.pc) * Neff;
    w.rWr = w.W + static_cast<size_t>(w.pc) * Neff;
    w.bytes = tile_bytes(w.pc, Neff);
    return w;
}

// What a scan of any number of variants can use (no more than kBlockM at a time), and what it can do with.
size_t wald_ws(int P, int Neff) { return carve_wald(nullptr, P, Neff, kBlockM, SIZE_MAX).bytes; }
size_t wald_least(int P, int Neff) { return std::min(wald_ws(P, Neff), tile_bytes(P, Neff)); }

}  // namespace

int flmm::wald_finish(const double* Gy, const double* Gs, const double* Gq, int nq, int64_t ldg, const double* rWr,
                      double var_df, int P, int n_real, int Mc, const int64_t* rows, double* f, double* beta, double* se,
                      double* sfve, int64_t ldo, double* max_F, cudaStream_t st) {
    const dim3 grid(ceil_div(Mc, kFinTile), ceil_div(P, kFinP));
    auto* k = nq > 0 ? k_wald_finish<true> : k_wald_finish<false>;
    k<<<grid, 256, 0, st>>>(Gy, Gs, Gq, nq, ldg, rWr, var_df, P, n_real, Mc, rows, f, beta, se, sfve, ldo, max_F);
    return check_launch("k_wald_finish");
}

extern "C" int flmm_wald_f64_workspace_bytes(int P, int Neff, size_t* bytes) {
    FLMM_REQUIRE(bytes && P >= 0 && Neff > 0, "flmm_wald_f64_workspace_bytes: bad arguments");
    *bytes = wald_ws(P, Neff);
    return FLMM_OK;
}

namespace {

// rows of [A | B] (rows, ka + kb) from A (rows, ka) and B (rows, kb)
__global__ void k_concat_rows(const double* __restrict__ A, int64_t lda, int ka, const double* __restrict__ B,
                              int64_t ldb, int kb, int rows, double* __restrict__ C) {
    const int k = ka + kb;
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (t >= static_cast<int64_t>(rows) * k) return;
    const int64_t r = t / k;
    const int c = static_cast<int>(t % k);
    C[t] = c < ka ? A[r * lda + c] : B[r * ldb + (c - ka)];
}

__global__ void k_spectrum_pad(const double* __restrict__ s, int k, int n0, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < k + n0) out[i] = i < k ? s[i] : 0.0;
}

// Column blocks outside, variant blocks inside.  A block's two products run on the tensor cores from digit planes
// (flmm_oz64.cu) where they are large enough, else in the fused FP64 tile kernel.
int wald_impl(const double* s, int Neff, const double* UYt, int64_t ldu, const double* log_delta, int P, int n_real,
              const double* USt, int64_t ldus, int Mc, const int64_t* rows, double* f, double* beta, double* se,
              double* sfve, int64_t ldo, double* max_F, double var_df, void* work, size_t work_bytes, cudaStream_t st) {
    const WaldWs w = carve_wald(work, P, Neff, Mc, work_bytes);
    int rc;
    for (int p0 = 0; p0 < P; p0 += w.pc) {
        const int pc = P - p0 < w.pc ? P - p0 : w.pc;
        const int nr = n_real > p0 ? (n_real - p0 < pc ? n_real - p0 : pc) : 0;
        double* W = w.A1 + static_cast<size_t>(pc) * Neff;
        k_wald_prep<<<ceil_div(static_cast<int64_t>(pc) * 32, 256), 256, 0, st>>>(s, Neff, UYt + p0 * ldu, ldu,
                                                                                 log_delta + p0, pc, W, w.A1, w.rWr);
        if ((rc = check_launch("k_wald_prep"))) return rc;
        auto out = [&](double* x) { return x ? x + p0 : x; };
        if (!w.tensor || !oz_worth(pc, Mc < w.mc ? Mc : w.mc, Neff)) {
            const dim3 grid(ceil_div(Mc, TM), ceil_div(pc, TP));
            k_wald_f64<<<grid, NT, 0, st>>>(W, w.A1, w.rWr, Neff, var_df, pc, nr, USt, ldus, Mc, rows, out(f), out(beta),
                                            out(se), out(sfve), ldo, max_F + p0);
            if ((rc = check_launch("k_wald_f64"))) return rc;
            continue;
        }
        if (p0 == 0 && (rc = oz_balance(USt, ldus, Mc, Neff, w.bal, st))) return rc;
        const OzOperand cols = oz_carve(w.cols, pc, Neff, 2, kOzRowsA);
        if ((rc = oz_digits(cols, 0, w.A1, Neff, false, w.bal, 1, st))) return rc;
        if ((rc = oz_digits(cols, 1, W, Neff, false, w.bal, 2, st))) return rc;
        for (int m0 = 0; m0 < Mc; m0 += w.mc) {
            const int mc = Mc - m0 < w.mc ? Mc - m0 : w.mc;
            const double* US = USt + m0 * ldus;
            const OzOperand vars = oz_carve(w.vars, mc, Neff, 2, kOzRowsB);
            if ((rc = oz_digits(vars, 0, US, ldus, false, w.bal, -1, st))) return rc;
            if ((rc = oz_digits(vars, 1, US, ldus, true, w.bal, -2, st))) return rc;
            const int64_t gs = static_cast<int64_t>(pc) * mc;
            const OzProduct prod{w.A1, Neff, static_cast<int64_t>(pc) * Neff, US, ldus, {false, true},
                                 OzGate::kBalanced, w.G, mc, gs, nullptr, 0};
            if ((rc = oz_gemm(cols, vars, prod, st))) return rc;
            if ((rc = wald_finish(w.G, w.G + gs, nullptr, 0, mc, w.rWr, var_df, pc, nr, mc, rows ? rows + m0 : rows, out(f),
                                  out(beta), out(se), out(sfve), ldo, max_F + p0, st)))
                return rc;
        }
    }
    return FLMM_OK;
}

size_t lowrank_cat_doubles(int k, int N, int P, int Mc) {
    return static_cast<size_t>(k + N) * (1 + static_cast<size_t>(P) + static_cast<size_t>(Mc));
}

}  // namespace

extern "C" int flmm_wald_f64(const double* s, int Neff, const double* UYt, int64_t ldu, const double* log_delta, int P,
                             int n_real, const double* USt, int64_t ldus, int Mc, const int64_t* rows, double* f,
                             double* beta, double* se, double* sfve, int64_t ldo, double* max_F, void* work,
                             size_t work_bytes, void* stream) {
    FLMM_REQUIRE(s && UYt && log_delta && max_F && work && Neff > 1 && P >= 0 && Mc >= 0 && ldu >= Neff &&
                     ldus >= Neff && n_real >= 0 && n_real <= P,
                 "flmm_wald_f64: bad arguments");
    FLMM_REQUIRE(n_real == 0 || Mc == 0 || (rows && f && beta && se && sfve && ldo >= n_real),
                 "flmm_wald_f64: real-column outputs missing");
    FLMM_REQUIRE(Mc == 0 || USt, "flmm_wald_f64: USt is NULL");
    if (work_bytes < wald_least(P, Neff))
        return fail(FLMM_ERR_WORKSPACE, "flmm_wald_f64: need %zu bytes, got %zu", wald_least(P, Neff), work_bytes);
    if (P == 0 || Mc == 0) return FLMM_OK;
    return wald_impl(s, Neff, UYt, ldu, log_delta, P, n_real, USt, ldus, Mc, rows, f, beta, se, sfve, ldo, max_F,
                     static_cast<double>(Neff - 1), work, work_bytes, as_stream(stream));
}

extern "C" int flmm_wald_lowrank_f64_workspace_bytes(int k, int N, int P, int Mc, size_t* bytes) {
    FLMM_REQUIRE(bytes && k > 0 && N > 0 && P >= 0 && Mc >= 0, "flmm_wald_lowrank_f64_workspace_bytes: bad arguments");
    *bytes = sizeof(double) * lowrank_cat_doubles(k, N, P, Mc) + 256 + wald_ws(P, k + N);
    return FLMM_OK;
}

extern "C" int flmm_wald_lowrank_f64(const double* s, int k, const double* UYt, int64_t ldu, const double* UUYt,
                                     int64_t lduu, int N, int Neff, const double* log_delta, int P, int n_real,
                                     const double* USt, int64_t ldus, const double* UUSt, int64_t lduus, int Mc,
                                     const int64_t* rows, double* f, double* beta, double* se, double* sfve,
                                     int64_t ldo, double* max_F, void* work, size_t work_bytes, void* stream) {
    FLMM_REQUIRE(s && UYt && UUYt && log_delta && max_F && work && k > 0 && N > 0 && Neff > 1 && P >= 0 && Mc >= 0 &&
                     ldu >= k && lduu >= N && ldus >= k && lduus >= N && n_real >= 0 && n_real <= P,
                 "flmm_wald_lowrank_f64: bad arguments");
    FLMM_REQUIRE(n_real == 0 || Mc == 0 || (rows && f && beta && se && sfve && ldo >= n_real),
                 "flmm_wald_lowrank_f64: real-column outputs missing");
    FLMM_REQUIRE(Mc == 0 || (USt && UUSt), "flmm_wald_lowrank_f64: variant operands missing");
    const size_t cat = sizeof(double) * lowrank_cat_doubles(k, N, P, Mc), need = cat + 256 + wald_least(P, k + N);
    if (work_bytes < need)
        return fail(FLMM_ERR_WORKSPACE, "flmm_wald_lowrank_f64: need %zu bytes, got %zu", need, work_bytes);
    if (P == 0 || Mc == 0) return FLMM_OK;
    // The off-rank directions enter every form with weight 1 / delta, i.e. as eigen-directions with s = 0: the scan
    // is the compat scan over [on-rank | off-rank] = k + N directions with var_df = Neff - 1
    // (fasterlmm/lowrank.py:274-299).
    cudaStream_t st = as_stream(stream);
    const int kc = k + N;
    double* s_cat = static_cast<double*>(work);
    double* UY_cat = s_cat + kc;
    double* US_cat = UY_cat + static_cast<size_t>(P) * kc;
    const size_t at = (cat + 255) / 256 * 256;
    void* rest = reinterpret_cast<char*>(work) + at;
    k_spectrum_pad<<<ceil_div(kc, 256), 256, 0, st>>>(s, k, N, s_cat);
    int rc = check_launch("k_spectrum_pad");
    if (rc) return rc;
    k_concat_rows<<<ceil_div(static_cast<int64_t>(P) * kc, 256), 256, 0, st>>>(UYt, ldu, k, UUYt, lduu, N, P, UY_cat);
    if ((rc = check_launch("k_concat_rows"))) return rc;
    k_concat_rows<<<ceil_div(static_cast<int64_t>(Mc) * kc, 256), 256, 0, st>>>(USt, ldus, k, UUSt, lduus, N, Mc,
                                                                                 US_cat);
    if ((rc = check_launch("k_concat_rows"))) return rc;
    return wald_impl(s_cat, kc, UY_cat, kc, log_delta, P, n_real, US_cat, kc, Mc, rows, f, beta, se, sfve, ldo, max_F,
                     static_cast<double>(Neff - 1), rest, work_bytes - at, st);
}
