// Plain GLS form of the scan (fasterlmm/core.py:89-375), in FP64: the covariates stay in the model, so every
// delta needs the (C, C) Gram A = X~^T W X~ and its Cholesky, and every test carries the quadratic form
// B^T A^-1 B with B = X~^T W s.
//
//   * grid losses: A_g, its Cholesky and log det once per grid node (k_gls_grid_prep); per (node, column) the
//     weighted products u = X~^T W y and yWy (k_gls_grid_loss); first argmin per column (k_gls_argmin);
//   * per-column evaluations (golden section, the per-phenotype loss): one warp forms the Gram of the augmented
//     columns [X~ | y] at the column's own delta in a few passes over the samples, then one lane factors it;
//   * Wald: per column the null fit (A, beta_x, r, rWr) and the left operands w o r, w o x_c, w (k_gls_wald_prep),
//     then a tiled kernel accumulates num = (w o r)^T s, B_c = (w o x_c)^T s and sWs = w^T (s o s) per (column,
//     variant) and runs the reference's epilogue (k_gls_wald).
// Loss formulas and golden-section updates use non-contracting FP64 intrinsics in the reference's order; sums over
// samples are warp / tile sums, so refined log delta agrees with the reference to its FP64 noise.
#include <math.h>

#include "flmm_common.cuh"
#include "flmm_oz64.cuh"
#include "flmm_tc.cuh"

using namespace flmm;

namespace {

constexpr int kMaxGlsC = 30;                       // covariate columns supported by the GLS kernels
constexpr double kLog2Pi = 1.8378770664093453;     // log(2 pi) in FP64
constexpr int kPairChunk = 8;                      // weighted products accumulated per pass over the samples
constexpr int kEvalWarps = 4;                      // warps per block of the per-column evaluation kernels

// -2 log L from yWy, uAu, sum log(s + delta) and log det A (fasterlmm/core.py:180-186 / 216-222)
__device__ double gls_loss(double yWy, double uAu, double sum_log_sd, double logdet_a, int N, int C, bool reml) {
    const double rWr = fmax(add_rn(yWy, -uAu), kPosFloor);
    if (reml) {
        const double nc = static_cast<double>(N - C);
        const double t = add_rn(add_rn(kLog2Pi, log(rWr / nc)), 1.0);
        return add_rn(add_rn(mul_rn(nc, t), sum_log_sd), logdet_a);
    }
    const double n = static_cast<double>(N);
    const double t = add_rn(add_rn(kLog2Pi, log(rWr / n)), 1.0);
    return add_rn(mul_rn(n, t), sum_log_sd);
}

// In-place lower Cholesky of the row-major (C, C) matrix A (lower triangle read).  False when a pivot is not
// positive, where torch.linalg.cholesky_ex reports info > 0; the caller then uses the identity, as the reference does.
__device__ bool chol_lower(double* A, int C) {
    for (int j = 0; j < C; ++j) {
        double d = A[j * C + j];
        for (int k = 0; k < j; ++k) d -= A[j * C + k] * A[j * C + k];
        if (!(d > 0.0)) return false;
        d = sqrt(d);
        A[j * C + j] = d;
        for (int i = j + 1; i < C; ++i) {
            double v = A[i * C + j];
            for (int k = 0; k < j; ++k) v -= A[i * C + k] * A[j * C + k];
            A[i * C + j] = v / d;
        }
    }
    for (int i = 0; i < C; ++i)
        for (int j = i + 1; j < C; ++j) A[i * C + j] = 0.0;
    return true;
}

__device__ void set_identity(double* A, int C) {
    for (int i = 0; i < C; ++i)
        for (int j = 0; j < C; ++j) A[i * C + j] = (i == j) ? 1.0 : 0.0;
}

// z = L^-1 b in place (forward substitution), L row-major lower
__device__ void forward_solve(const double* L, int C, double* z) {
    for (int i = 0; i < C; ++i) {
        double v = z[i];
        for (int k = 0; k < i; ++k) v -= L[i * C + k] * z[k];
        z[i] = v / L[i * C + i];
    }
}

// x = L^-T z in place (back substitution)
__device__ void back_solve(const double* L, int C, double* x) {
    for (int i = C - 1; i >= 0; --i) {
        double v = x[i];
        for (int k = i + 1; k < C; ++k) v -= L[k * C + i] * x[k];
        x[i] = v / L[i * C + i];
    }
}

// Weighted Gram of the augmented columns a_0..a_C = (x~_0 .. x~_{C-1}, y) at one delta, by one warp:
// Gs[i * (C + 1) + j] = sum_n a_i[n] a_j[n] / (s[n] + delta) for j <= i, over the lane's samples first, first + step, ...
// Returns sum_n log(s[n] + delta).
__device__ double warp_gram(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx, int C,
                            const double* __restrict__ y, double delta, double* Gs, int first, int step) {
    const int lane = threadIdx.x & 31;
    const int K = C + 1;
    const int pairs = K * (K + 1) / 2;
    double sl = 0.0;
    int i0 = 0, j0 = 0;  // pair at the start of the chunk
    for (int q0 = 0; q0 < pairs; q0 += kPairChunk) {
        int pi[kPairChunk], pj[kPairChunk];
        int i = i0, j = j0;
#pragma unroll
        for (int k = 0; k < kPairChunk; ++k) {
            pi[k] = i;
            pj[k] = j;
            if (j < i) { ++j; } else { ++i; j = 0; }
        }
        i0 = i;
        j0 = j;
        double acc[kPairChunk] = {};
        for (int n = first; n < N; n += step) {
            const double sd = s[n] + delta;
            const double w = 1.0 / sd;
            if (q0 == 0) sl += log(sd);
#pragma unroll
            for (int k = 0; k < kPairChunk; ++k) {
                if (q0 + k < pairs) {
                    const double ai = pi[k] < C ? Xrt[pi[k] * ldx + n] : y[n];
                    const double aj = pj[k] < C ? Xrt[pj[k] * ldx + n] : y[n];
                    acc[k] += mul_rn(mul_rn(w, ai), aj);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kPairChunk; ++k) {
            const double v = warp_sum(acc[k]);
            if (lane == 0 && q0 + k < pairs) Gs[pi[k] * K + pj[k]] = v;
        }
    }
    __syncwarp();
    return warp_sum(sl);
}

// -2 log L from the augmented Gram Gs and sum log(s + delta), by one thread; A is scratch (C * C) and z (C).
__device__ double gram_loss(const double* Gs, double sum_log, int N, int C, bool reml, double* A, double* z) {
    const int K = C + 1;
    for (int i = 0; i < C; ++i) {
        for (int j = 0; j <= i; ++j) A[i * C + j] = Gs[i * K + j];
        z[i] = Gs[C * K + i];
    }
    const bool ok = chol_lower(A, C);
    if (!ok) set_identity(A, C);
    double logdet = 0.0;
    if (reml) {
        for (int i = 0; i < C; ++i) logdet += log(A[i * C + i]);
        logdet = 2.0 * logdet;
    }
    forward_solve(A, C, z);
    double uAu = 0.0;
    for (int i = 0; i < C; ++i) uAu += z[i] * z[i];
    return ok ? gls_loss(Gs[C * K + C], uAu, sum_log, logdet, N, C, reml) : INFINITY;
}

// One column's -2 log L at its own delta (fasterlmm/core.py:190-224), by one warp; A is per-warp scratch (C * C)
// and z (C).
__device__ double warp_pheno_loss(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx,
                                  int C, const double* __restrict__ y, double ld, bool reml, double* Gs, double* A,
                                  double* z) {
    const int lane = threadIdx.x & 31;
    const double sum_log = warp_gram(s, N, Xrt, ldx, C, y, exp(ld), Gs, lane, 32);
    double loss = 0.0;
    if (lane == 0) loss = gram_loss(Gs, sum_log, N, C, reml, A, z);
    __syncwarp();
    return __shfl_sync(0xffffffffu, loss, 0);
}

// ---- grid ----------------------------------------------------------------------------------------------------

// Per grid node g (one block): W[g, n] = 1 / (s[n] + delta_g), sum log(s + delta_g), A_g, its Cholesky L_g (identity
// and bad[g] = 1 when it fails) and log det A_g.
__global__ void k_gls_grid_prep(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx,
                                int C, const double* __restrict__ grid, double* __restrict__ W,
                                double* __restrict__ sum_log, double* __restrict__ Lg, double* __restrict__ logdet,
                                int32_t* __restrict__ bad) {
    __shared__ double A[kMaxGlsC * kMaxGlsC];
    __shared__ double red[32];
    const int g = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const double delta = exp(grid[g]);
    double sl = 0.0;
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
        const double sd = s[n] + delta;
        W[static_cast<int64_t>(g) * N + n] = 1.0 / sd;
        sl += log(sd);
    }
    sl = warp_sum(sl);
    if (lane == 0) red[warp] = sl;
    __syncthreads();  // W row complete
    const double* w = W + static_cast<int64_t>(g) * N;
    const int pairs = C * (C + 1) / 2;
    for (int q = warp; q < pairs; q += nwarps) {
        int i = 0, r = q;
        while (r > i) { r -= i + 1; ++i; }
        const int j = r;
        double acc = 0.0;
        for (int n = lane; n < N; n += 32) acc += mul_rn(mul_rn(w[n], Xrt[i * ldx + n]), Xrt[j * ldx + n]);
        acc = warp_sum(acc);
        if (lane == 0) A[i * C + j] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < nwarps; ++k) t += red[k];
        sum_log[g] = t;
        const bool ok = chol_lower(A, C);
        if (!ok) set_identity(A, C);
        double ld = 0.0;
        for (int i = 0; i < C; ++i) ld += log(A[i * C + i]);
        logdet[g] = 2.0 * ld;
        bad[g] = ok ? 0 : 1;
        double* L = Lg + static_cast<int64_t>(g) * C * C;
        for (int i = 0; i < C * C; ++i) L[i] = A[i];
    }
}

// loss[g, p] (fasterlmm/core.py:148-187): one warp per (g, column), u_c = sum_n W[g, n] x~_c[n] y[n] in chunks
__global__ void k_gls_grid_loss(const double* __restrict__ W, const double* __restrict__ Xrt, int64_t ldx, int C,
                                const double* __restrict__ Yrt, int64_t ldy, int N, int P,
                                const double* __restrict__ sum_log, const double* __restrict__ Lg,
                                const double* __restrict__ logdet, const int32_t* __restrict__ bad, int reml,
                                double* __restrict__ loss) {
    __shared__ double zs[kEvalWarps][kMaxGlsC + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.y;
    const int64_t p = static_cast<int64_t>(blockIdx.x) * kEvalWarps + warp;
    if (p >= P) return;
    const double* w = W + static_cast<int64_t>(g) * N;
    const double* y = Yrt + p * ldy;
    double* z = zs[warp];
    for (int c0 = 0; c0 <= C; c0 += kPairChunk) {
        double acc[kPairChunk] = {};
        for (int n = lane; n < N; n += 32) {
            const double yy = mul_rn(y[n], y[n]);  // yWy = w @ (Y o Y), fasterlmm/core.py:177
#pragma unroll
            for (int k = 0; k < kPairChunk; ++k) {
                const int c = c0 + k;
                if (c < C) acc[k] += mul_rn(mul_rn(w[n], Xrt[c * ldx + n]), y[n]);
                else if (c == C) acc[k] += mul_rn(w[n], yy);
            }
        }
#pragma unroll
        for (int k = 0; k < kPairChunk; ++k) {
            const double v = warp_sum(acc[k]);
            if (lane == 0 && c0 + k <= C) z[c0 + k] = v;
        }
    }
    __syncwarp();
    if (lane == 0) {
        const double yWy = z[C];
        forward_solve(Lg + static_cast<int64_t>(g) * C * C, C, z);
        double uAu = 0.0;
        for (int i = 0; i < C; ++i) uAu += z[i] * z[i];
        loss[static_cast<int64_t>(g) * P + p] =
            bad[g] ? INFINITY : gls_loss(yWy, uAu, sum_log[g], logdet[g], N, C, reml != 0);
    }
}

// first argmin over g of loss (G, P), as torch.argmin
__global__ void k_gls_argmin(const double* __restrict__ loss, int G, int P, int32_t* __restrict__ idx) {
    const int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (p >= P) return;
    double best = loss[p];
    int bi = 0;
    for (int g = 1; g < G; ++g) {
        const double v = loss[static_cast<int64_t>(g) * P + p];
        if (v < best) { best = v; bi = g; }
    }
    idx[p] = bi;
}

// ---- per-column evaluations -----------------------------------------------------------------------------------

__device__ __forceinline__ size_t eval_smem_doubles(int C) {
    return static_cast<size_t>(C + 1) * (C + 1) + static_cast<size_t>(C) * C + (C + 1);
}

// loss[p] at log_delta[p], one warp per column
__global__ void k_gls_pheno_loss(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx,
                                 int C, const double* __restrict__ Yrt, int64_t ldy, int P,
                                 const double* __restrict__ ld, int reml, double* __restrict__ loss) {
    extern __shared__ double sm[];
    const int warp = threadIdx.x >> 5;
    const int64_t p = static_cast<int64_t>(blockIdx.x) * kEvalWarps + warp;
    if (p >= P) return;
    double* Gs = sm + warp * eval_smem_doubles(C);
    double* A = Gs + (C + 1) * (C + 1);
    double* z = A + C * C;
    const double v = warp_pheno_loss(s, N, Xrt, ldx, C, Yrt + p * ldy, ld[p], reml != 0, Gs, A, z);
    if ((threadIdx.x & 31) == 0) loss[p] = v;
}

// golden-section search on [grid[i-1], grid[i+1]], one warp per column (fasterlmm/core.py:245-264)
__global__ void k_gls_golden(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx, int C,
                             const double* __restrict__ Yrt, int64_t ldy, int P, const double* __restrict__ grid,
                             int G, const int32_t* __restrict__ idx, int refine, int reml, double lo, double hi,
                             double* __restrict__ log_delta) {
    extern __shared__ double sm[];
    const int warp = threadIdx.x >> 5;
    const int64_t p = static_cast<int64_t>(blockIdx.x) * kEvalWarps + warp;
    if (p >= P) return;
    const int i = idx[p];
    if (!refine) {
        if ((threadIdx.x & 31) == 0) log_delta[p] = grid[i];
        return;
    }
    double* Gs = sm + warp * eval_smem_doubles(C);
    double* A = Gs + (C + 1) * (C + 1);
    double* z = A + C * C;
    const double* y = Yrt + p * ldy;
    const bool rm = reml != 0;
    double a = grid[max(i - 1, 0)], b = grid[min(i + 1, G - 1)];
    const double inv_phi = 2.0 / (1.0 + sqrt(5.0));
    const double inv_phi2 = mul_rn(inv_phi, inv_phi);
    double c = add_rn(a, mul_rn(inv_phi2, add_rn(b, -a)));
    double d = add_rn(a, mul_rn(inv_phi, add_rn(b, -a)));
    double fc = warp_pheno_loss(s, N, Xrt, ldx, C, y, c, rm, Gs, A, z);
    double fd = warp_pheno_loss(s, N, Xrt, ldx, C, y, d, rm, Gs, A, z);
    for (int it = 0; it < 50; ++it) {
        const bool cond = fc < fd;
        b = cond ? d : b;
        a = cond ? a : c;
        c = add_rn(a, mul_rn(inv_phi2, add_rn(b, -a)));
        d = add_rn(a, mul_rn(inv_phi, add_rn(b, -a)));
        if (it == 49) break;  // the last bracket is not compared again
        fc = warp_pheno_loss(s, N, Xrt, ldx, C, y, c, rm, Gs, A, z);
        fd = warp_pheno_loss(s, N, Xrt, ldx, C, y, d, rm, Gs, A, z);
    }
    if ((threadIdx.x & 31) == 0) log_delta[p] = fmin(fmax(mul_rn(0.5, add_rn(a, b)), lo), hi);
}

// The same search with a cluster of two blocks per column, one for each evaluation of a step: the FP64 pipe of an SM bounds
// a step, and a study of tens of columns leaves most SMs idle otherwise.  A block's threads form the weights (one division
// per eigenvalue; a warp of k_gls_golden forms them again for every eight products of its Gram) and logarithms into shared
// memory, its warps add the Gram's products four at a time, each sum in the order of k_gls_golden's lanes and butterfly, so
// every loss keeps its bits; thread 0 puts the loss into both blocks, and both carry the search.  A point that is, to the
// bit, one of the step before keeps its loss.  60 columns x 300 samples, C = 5, with the grid: 7.5 ms with a warp per column,
// 2.3 with one block, 1.5 here.  Beyond ~12,000 samples the weights no longer fit in shared memory and k_gls_golden runs.
constexpr int kBlockThreads = 256;
constexpr int kBlockPairs = 4;
constexpr size_t kBlockSmemMax = 200 * 1024;

size_t golden_block_smem(int N, int C) {
    return sizeof(double) * (2 * static_cast<size_t>(N) + static_cast<size_t>(C + 1) * (C + 1) + static_cast<size_t>(C) * C +
                             (C + 1));
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBlockThreads)
k_gls_golden_block(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx, int C,
                   const double* __restrict__ Yrt, int64_t ldy, const double* __restrict__ grid, int G,
                   const int32_t* __restrict__ idx, int reml, double lo, double hi, double* __restrict__ log_delta) {
    extern __shared__ double sm[];
    __shared__ double delta_s, log_s, loss_s[2][2];  // loss_s[step % 2][evaluation]
    __shared__ int kept_s;
    const int64_t p = blockIdx.x >> 1;
    const int my_e = static_cast<int>(tc::cluster_ctarank());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = C + 1, pairs = K * (K + 1) / 2;
    double* w = sm;        // [N]
    double* lg = w + N;    // [N]
    double* Gs = lg + N;   // Gram, then the factor and a vector
    const double* y = Yrt + p * ldy;
    Bracket br(grid, G, idx[p]);
    const int groups = (pairs + kBlockPairs - 1) / kBlockPairs;  // of products; one more sum is the logarithms'
    tc::cluster_sync();  // the other block runs: its shared memory may be written
    for (int it = 0; it < 50; ++it) {
        double kept_loss = 0.0;
        if (tid == 0) {
            kept_s = it > 0 && br.narrow_kept(loss_s[(it - 1) & 1], my_e, &kept_loss);
            delta_s = exp(my_e ? br.d() : br.c());
        }
        __syncthreads();
        const bool kept = kept_s != 0;
        if (!kept) {
            for (int n = tid; n < N; n += kBlockThreads) {
                const double sd = s[n] + delta_s;
                w[n] = 1.0 / sd;
                lg[n] = log(sd);
            }
            __syncthreads();
            for (int q = warp; q <= groups; q += kBlockThreads / 32) {
                if (q == groups) {
                    double sl = 0.0;
                    for (int n = lane; n < N; n += 32) sl += lg[n];
                    sl = warp_sum(sl);
                    if (lane == 0) log_s = sl;
                    continue;
                }
                const double *ai[kBlockPairs], *aj[kBlockPairs];
                int at[kBlockPairs];
#pragma unroll
                for (int k = 0; k < kBlockPairs; ++k) {
                    const int r = min(q * kBlockPairs + k, pairs - 1);
                    int pi = static_cast<int>((sqrtf(8.0f * r + 1.0f) - 1.0f) * 0.5f);
                    if (pi * (pi + 1) / 2 > r) --pi;
                    if ((pi + 1) * (pi + 2) / 2 <= r) ++pi;
                    const int pj = r - pi * (pi + 1) / 2;
                    at[k] = pi * K + pj;
                    ai[k] = pi < C ? Xrt + pi * ldx : y;
                    aj[k] = pj < C ? Xrt + pj * ldx : y;
                }
                double acc[kBlockPairs] = {};
                for (int n = lane; n < N; n += 32) {
                    const double wn = w[n];
                    double wa = 0.0;
#pragma unroll
                    for (int k = 0; k < kBlockPairs; ++k) {
                        if (k == 0 || ai[k] != ai[k - 1]) wa = mul_rn(wn, ai[k][n]);
                        acc[k] += mul_rn(wa, aj[k][n]);
                    }
                }
#pragma unroll
                for (int k = 0; k < kBlockPairs; ++k) {
                    const double v = warp_sum(acc[k]);
                    if (lane == 0 && q * kBlockPairs + k < pairs) Gs[at[k]] = v;
                }
            }
            __syncthreads();
        }
        if (tid == 0) {
            const double loss = kept ? kept_loss : gram_loss(Gs, log_s, N, C, reml != 0, Gs + K * K, Gs + K * K + C * C);
            const uint32_t at = tc::smem_u32(&loss_s[it & 1][my_e]);
#pragma unroll
            for (uint32_t r = 0; r < 2; ++r)
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(tc::map_to_rank(at, r)), "d"(loss) : "memory");
        }
        // (two buffers: a block can be one step ahead of the other's read, not two; and after the last step neither leaves
        // before the other has written)
        tc::cluster_sync();
    }
    if (tid == 0 && my_e == 0) {
        const double* loss = loss_s[49 & 1];
        br.narrow(loss[0] < loss[1]);
        log_delta[p] = fmin(fmax(mul_rn(0.5, add_rn(br.a, br.b)), lo), hi);
    }
}

// ---- Wald ------------------------------------------------------------------------------------------------------

// Null fit of column p at its log delta (fasterlmm/core.py:328-341): A_p, L_p (identity when the Cholesky fails),
// beta_x = A^-1 u, r = y~ - X~ beta_x, rWr = sum w r^2, and the left operands of the scan, rows of N entries: w o r at
// Rv, w at Wv (column pitch rv_stride), and C rows at Qv (column pitch qv_stride): w o x~_c, or with `solved` the rows
// of L^-1 X~^T W, whose products with a variant are the terms of B^T A^-1 B as squares.  A block a column: a warp's
// chains of FP64 operations are slow on this pipe, so four share a column's samples (660 columns x 800 samples, C = 5: 0.28
// ms with four columns a block, a warp each, 0.24 with one; 0.18 here).
constexpr int kPrepThreads = 128;

__global__ void __launch_bounds__(kPrepThreads)
k_gls_wald_prep(const double* __restrict__ s, int N, const double* __restrict__ Xrt, int64_t ldx, int C,
                const double* __restrict__ Yrt, int64_t ldy, const double* __restrict__ ld, int solved,
                double* __restrict__ Rv, double* __restrict__ Wv, int64_t rv_stride, double* __restrict__ Qv,
                int64_t qv_stride, double* __restrict__ Lp, double* __restrict__ rWr) {
    extern __shared__ double sm[];
    __shared__ double red[kPrepThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, K = C + 1;
    const int64_t p = blockIdx.x;
    double* Gs = sm;  // a Gram of each warp's samples, added into the first
    double* A = Gs + (kPrepThreads / 32) * K * K;
    double* z = A + C * C;
    const double* y = Yrt + p * ldy;
    const double delta = exp(ld[p]);
    warp_gram(s, N, Xrt, ldx, C, y, delta, Gs + warp * K * K, tid, kPrepThreads);
    __syncthreads();
    for (int e = tid; e < K * K; e += kPrepThreads)
        if (e % K <= e / K)
            for (int w = 1; w < kPrepThreads / 32; ++w) Gs[e] += Gs[w * K * K + e];
    __syncthreads();
    if (tid == 0) {
        for (int i = 0; i < C; ++i) {
            for (int j = 0; j <= i; ++j) A[i * C + j] = Gs[i * K + j];
            z[i] = Gs[C * K + i];
        }
        if (!chol_lower(A, C)) set_identity(A, C);
        forward_solve(A, C, z);
        back_solve(A, C, z);  // z = beta_x
        if (solved) {
            for (int i = 0; i < C; ++i) Gs[i] = 1.0 / A[i * C + i];
        } else {
            double* L = Lp + p * C * C;
            for (int i = 0; i < C * C; ++i) L[i] = A[i];
        }
    }
    __syncthreads();
    double* rv = Rv + p * rv_stride;
    double* wv = Wv + p * rv_stride;
    double acc = 0.0;
    for (int n = tid; n < N; n += kPrepThreads) {
        const double w = 1.0 / (s[n] + delta);
        double fit = 0.0;
        for (int c = 0; c < C; ++c) fit = fma(Xrt[c * ldx + n], z[c], fit);
        const double r = add_rn(y[n], -fit);
        const double wr = mul_rn(w, r);
        acc += mul_rn(wr, r);
        rv[n] = wr;
        double* col = Qv + p * qv_stride + n;  // this sample's entries of the C rows, N apart
        for (int c = 0; c < C; ++c) {
            double v = mul_rn(w, Xrt[c * ldx + n]);
            if (solved) {
                for (int k = 0; k < c; ++k) v = fma(-A[c * C + k], col[static_cast<int64_t>(k) * N], v);
                v = mul_rn(v, Gs[c]);
            }
            col[static_cast<int64_t>(c) * N] = v;
        }
        wv[n] = w;
    }
    acc = warp_sum(acc);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kPrepThreads / 32; ++w) acc += red[w];
        rWr[p] = acc;
    }
}

constexpr int WP = 16, WM = 16, WK = 8, WT = 256;

// Tile of 16 columns x 16 variants, thread = one (column, variant): num, B_0..B_{C-1} in acc[0..C] and sWs in
// acc[KOPS - 1], accumulated over the samples in chunks of 8, then fasterlmm/core.py:346-371 on the sums.
// KOPS >= C + 2 is the register budget (8, 16 or 32 operands).
template <int KOPS>
__global__ void __launch_bounds__(WT)
k_gls_wald(const double* __restrict__ Lv, const double* __restrict__ Lp, const double* __restrict__ rWr, int N,
           int C, int P, int n_real, const double* __restrict__ Srt, int64_t lds, int M,
           const int64_t* __restrict__ rows, double* __restrict__ f, double* __restrict__ beta, double* __restrict__ se,
           double* __restrict__ sfve, int64_t ldo, double* __restrict__ max_F) {
    extern __shared__ double sm[];
    const int nops = C + 2;
    double* Ls = sm;                                   // [WP][nops][WK]
    double* Ss = Ls + WP * nops * WK;                  // [WM][WK]
    const int tid = threadIdx.x;
    const int pi = tid >> 4, mi = tid & 15;            // 16 consecutive threads share a column
    const int p0 = blockIdx.y * WP, m0 = blockIdx.x * WM;
    const int p = p0 + pi, m = m0 + mi;
    double acc[KOPS];
#pragma unroll
    for (int k = 0; k < KOPS; ++k) acc[k] = 0.0;
    for (int n0 = 0; n0 < N; n0 += WK) {
        for (int t = tid; t < WP * nops * WK; t += WT) {
            const int q = t / (nops * WK), rem = t % (nops * WK), op = rem / WK, k = rem % WK;
            const int gp = p0 + q, gn = n0 + k;
            Ls[t] = (gp < P && gn < N) ? Lv[(static_cast<int64_t>(gp) * nops + op) * N + gn] : 0.0;
        }
        for (int t = tid; t < WM * WK; t += WT) {
            const int q = t / WK, k = t % WK;
            const int gm = m0 + q, gn = n0 + k;
            Ss[t] = (gm < M && gn < N) ? Srt[static_cast<int64_t>(gm) * lds + gn] : 0.0;
        }
        __syncthreads();
        const double* lrow = Ls + pi * nops * WK;
        const double* srow = Ss + mi * WK;
#pragma unroll
        for (int k = 0; k < WK; ++k) {
            const double sv = srow[k];
#pragma unroll
            for (int op = 0; op < KOPS - 1; ++op)
                if (op < C + 1) acc[op] = fma(lrow[op * WK + k], sv, acc[op]);
            acc[KOPS - 1] = fma(lrow[(C + 1) * WK + k], mul_rn(sv, sv), acc[KOPS - 1]);
        }
        __syncthreads();
    }
    double F = -INFINITY;
    if (p < P && m < M) {
        // quad = B^T A^-1 B = |L^-1 B|^2
        const double* L = Lp + static_cast<int64_t>(p) * C * C;
        double quad = 0.0;
#pragma unroll
        for (int i = 0; i < KOPS - 2; ++i) {
            if (i < C) {
                double v = acc[1 + i];
#pragma unroll
                for (int k = 0; k < KOPS - 2; ++k)
                    if (k < i) v -= L[i * C + k] * acc[1 + k];
                v = v / L[i * C + i];
                acc[1 + i] = v;
                quad += v * v;
            }
        }
        const double num = acc[0];
        const double denom = fmax(add_rn(acc[KOPS - 1], -quad), kPosFloor);
        const double b = num / denom;
        const double q = mul_rn(num, num);
        const double rwr = rWr[p];
        const double rss = fmax(add_rn(rwr, -(q / denom)), kPosFloor);
        const double var_b = (rss / static_cast<double>(N - C - 1)) / denom;
        F = mul_rn(b, b) / var_b;
        if (p < n_real) {
            const int64_t o = rows[m] * ldo + p;
            f[o] = F;
            beta[o] = b;
            se[o] = sqrt(var_b);
            sfve[o] = sqrt(fmax(q / mul_rn(denom, rwr), 0.0));
        }
    }
    // column max over this tile's 16 variants (a half-warp), NaN kept
    bool nan_f = isnan(F);
    double v = nan_f ? -INFINITY : F;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        nan_f |= __shfl_xor_sync(0xffffffffu, static_cast<int>(nan_f), o) != 0;
    }
    if (mi == 0 && p < P) {
        if (nan_f) v = NAN;
        if (v >= 0.0 || isnan(v)) atomic_max_nonneg(max_F + p, v);
    }
}

// Workspace of the grid stage: grid nodes, W (G, N), sum log, log det, L_g (G, C, C), bad (G), loss (G, P)
struct GridWs {
    double *grid, *W, *sum_log, *logdet, *Lg, *loss;
    int32_t* bad;
    size_t bytes;
};

GridWs carve_grid(void* base, int N, int C, int P, int G) {
    GridWs w{};
    size_t off = 0;
    const uintptr_t b = reinterpret_cast<uintptr_t>(base);
    auto take = [&](size_t nbytes) {
        const uintptr_t p = b + off;
        off += (nbytes + 255) / 256 * 256;
        return p;
    };
    w.grid = reinterpret_cast<double*>(take(sizeof(double) * G));  // (addresses only when base is non-null)
    w.W = reinterpret_cast<double*>(take(sizeof(double) * static_cast<size_t>(G) * N));
    w.sum_log = reinterpret_cast<double*>(take(sizeof(double) * G));
    w.logdet = reinterpret_cast<double*>(take(sizeof(double) * G));
    w.Lg = reinterpret_cast<double*>(take(sizeof(double) * static_cast<size_t>(G) * C * C));
    w.bad = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * G));
    w.loss = reinterpret_cast<double*>(take(sizeof(double) * static_cast<size_t>(G) * P));
    w.bytes = off;
    return w;
}

constexpr int kWaldChunk = 4096;  // columns prepared per pass of the FP64 tile kernel

// Blocks of the tensor-core path: (C + 2) operand rows per column, kBlockRows rows and kBlockM variants at most, fewer
// where their digit planes (16 bytes per element) would pass kPlaneBytes.  A shorter workspace gets smaller blocks, and the
// FP64 tile kernel's where the smallest do not fit.
constexpr int kBlockRows = 6144, kBlockM = 4096;
constexpr size_t kPlaneBytes = size_t(256) << 20;

struct WaldWs {
    bool tensor;
    int pc, mc;             // columns and variants of a block
    double *RW, *Q, *rWr;   // w o r and w (2, pc, N), L^-1 X~^T W (pc, C, N)
    double *G, *Gq;         // sums: num and sWs (2, pc, mc), the quadratic form's terms (pc, C, mc)
    char *rw_op, *q_op, *s_op;
    int* bal;               // balancing exponents and their scratch
    size_t bytes;
};

WaldWs carve_blocks(void* base, int N, int C, int columns, int variants) {
    WaldWs w{};
    w.tensor = true;
    w.pc = columns;
    w.mc = variants;
    size_t off = 0;
    const uintptr_t b0 = (reinterpret_cast<uintptr_t>(base) + 1023) / 1024 * 1024;
    auto take = [&](size_t n) {
        const uintptr_t p = b0 + off;
        off += (n + 1023) / 1024 * 1024;
        return p;
    };
    const size_t n = N, pc = w.pc, mc = w.mc;
    w.rWr = reinterpret_cast<double*>(take(sizeof(double) * pc));
    w.RW = reinterpret_cast<double*>(take(2 * sizeof(double) * pc * n));
    w.Q = reinterpret_cast<double*>(take(sizeof(double) * pc * C * n));
    w.G = reinterpret_cast<double*>(take(2 * sizeof(double) * pc * mc));
    w.Gq = reinterpret_cast<double*>(take(sizeof(double) * pc * C * mc));
    w.rw_op = reinterpret_cast<char*>(take(oz_operand_bytes(w.pc, N, 2, kOzRowsA)));
    w.q_op = reinterpret_cast<char*>(take(oz_operand_bytes(w.pc * C, N, 1, kOzRowsA)));
    w.s_op = reinterpret_cast<char*>(take(oz_operand_bytes(w.mc, N, 2, kOzRowsB)));
    w.bal = reinterpret_cast<int*>(take(sizeof(int) * oz_balance_ints(N)));
    w.bytes = off + 1024;
    return w;
}

// The FP64 tile kernel's workspace for pc columns: operands of (C + 2) rows, factors, rWr.
size_t tile_column_bytes(int N, int C) {
    return sizeof(double) * ((static_cast<size_t>(C) + 2) * N + static_cast<size_t>(C) * C + 1);
}
size_t tile_bytes(int N, int C, int P) { return tile_column_bytes(N, C) * (P < kWaldChunk ? P : kWaldChunk) + 1024; }

// The blocks of a scan of P columns x M variants in `bytes` of workspace (pc: columns of a pass also of the tile kernel).
WaldWs carve_wald(void* base, int N, int C, int P, int M, size_t bytes) {
    const size_t fit = kPlaneBytes / (16 * static_cast<size_t>(N));
    const size_t rows = fit < static_cast<size_t>(kBlockRows) ? fit : kBlockRows;
    int pc = static_cast<int>(rows / (C + 2));
    pc = pc < 1 ? 1 : (P < pc ? (P > 0 ? P : 1) : pc);
    int mc = static_cast<int>(fit / 2 < static_cast<size_t>(kBlockM) ? fit / 2 / kOzRowsB * kOzRowsB : kBlockM);
    mc = mc < kOzRowsB ? kOzRowsB : mc;
    const int most = (M > 0 ? (M - 1) / kOzRowsB + 1 : 1) * kOzRowsB;
    if (most < mc) mc = most;
    for (; oz_worth(static_cast<int64_t>(pc) * (C + 2), M < mc ? M : mc, N);) {
        const WaldWs w = carve_blocks(base, N, C, pc, mc);
        if (w.bytes <= bytes) return w;
        if (mc > 512 || (pc == 1 && mc > kOzRowsB)) mc = (mc / 2 + kOzRowsB - 1) / kOzRowsB * kOzRowsB;
        else if (pc > 1) pc = (pc + 1) / 2;
        else break;
    }
    WaldWs w{};
    w.mc = M;
    const size_t columns = bytes / tile_column_bytes(N, C);
    w.pc = P < kWaldChunk ? P : kWaldChunk;
    if (columns < static_cast<size_t>(w.pc)) w.pc = static_cast<int>(columns);
    w.bytes = tile_bytes(N, C, P);
    return w;
}

size_t wald_ws(int N, int C, int P) { return carve_wald(nullptr, N, C, P, kBlockM, SIZE_MAX).bytes; }
size_t wald_least(int N, int C, int P) {
    const size_t tiles = tile_bytes(N, C, P), full = wald_ws(N, C, P);
    return tiles < full ? tiles : full;
}

__global__ void k_shift_diagonal(double* __restrict__ A, int N, int64_t lda, double v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) A[static_cast<int64_t>(i) * lda + i] += v;
}

__global__ void k_clamp_nonneg(const double* __restrict__ x, int64_t n, double* __restrict__ y) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < n) y[i] = fmax(x[i], 0.0);
}

// (the kernels' limit is that of kMaxGlsC whatever the call's C: another host thread's call must not lower it)
size_t eval_smem_bytes(int C) {
    return sizeof(double) * kEvalWarps *
           (static_cast<size_t>(C + 1) * (C + 1) + static_cast<size_t>(C) * C + (C + 1));
}

int check_c(int C, const char* fn) {
    if (C < 1 || C > kMaxGlsC) return fail(FLMM_ERR_ARG, "%s: covariate columns must be in 1..%d", fn, kMaxGlsC);
    return FLMM_OK;
}

}  // namespace

extern "C" int flmm_gls_loss_workspace_bytes(int N, int C, int P, int n_ld, size_t* bytes) {
    FLMM_REQUIRE(bytes && N > 0 && C > 0 && P >= 0 && n_ld > 0, "flmm_gls_loss_workspace_bytes: bad arguments");
    *bytes = carve_grid(nullptr, N, C, P, n_ld).bytes;
    return FLMM_OK;
}

extern "C" int flmm_gls_loss_f64(const double* s, int N, const double* Xrt, int64_t ldx, int C, const double* Yrt,
                                 int64_t ldy, int P, const double* log_delta, int n_ld, int per_column, int reml,
                                 double* loss, void* work, size_t work_bytes, void* stream) {
    FLMM_REQUIRE(s && Xrt && Yrt && log_delta && loss && N > C && ldx >= N && ldy >= N && P >= 0 && n_ld > 0,
                 "flmm_gls_loss_f64: bad arguments");
    int rc = check_c(C, "flmm_gls_loss_f64");
    if (rc) return rc;
    if (P == 0) return FLMM_OK;
    cudaStream_t st = as_stream(stream);
    const size_t smem = eval_smem_bytes(C);
    if (per_column) {
        FLMM_REQUIRE(n_ld == P, "flmm_gls_loss_f64: per-column mode needs one log delta per column");
        FLMM_CUDA(cudaFuncSetAttribute(k_gls_pheno_loss, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)eval_smem_bytes(kMaxGlsC)));
        k_gls_pheno_loss<<<ceil_div(P, kEvalWarps), 32 * kEvalWarps, smem, st>>>(s, N, Xrt, ldx, C, Yrt, ldy, P,
                                                                                  log_delta, reml, loss);
        return check_launch("k_gls_pheno_loss");
    }
    FLMM_REQUIRE(work, "flmm_gls_loss_f64: grid mode needs a workspace");
    GridWs ws = carve_grid(work, N, C, P, n_ld);
    if (work_bytes < ws.bytes)
        return fail(FLMM_ERR_WORKSPACE, "flmm_gls_loss_f64: need %zu bytes, got %zu", ws.bytes, work_bytes);
    k_gls_grid_prep<<<n_ld, 256, 0, st>>>(s, N, Xrt, ldx, C, log_delta, ws.W, ws.sum_log, ws.Lg, ws.logdet, ws.bad);
    if ((rc = check_launch("k_gls_grid_prep"))) return rc;
    dim3 grid(ceil_div(P, kEvalWarps), n_ld);
    k_gls_grid_loss<<<grid, 32 * kEvalWarps, 0, st>>>(ws.W, Xrt, ldx, C, Yrt, ldy, N, P, ws.sum_log, ws.Lg, ws.logdet,
                                                       ws.bad, reml, loss);
    return check_launch("k_gls_grid_loss");
}

extern "C" int flmm_fit_delta_gls_workspace_bytes(int N, int C, int P, int n_grid, size_t* bytes) {
    FLMM_REQUIRE(bytes && N > 0 && C > 0 && P >= 0 && n_grid > 0, "flmm_fit_delta_gls_workspace_bytes: bad arguments");
    *bytes = carve_grid(nullptr, N, C, P, n_grid).bytes;
    return FLMM_OK;
}

extern "C" int flmm_fit_delta_gls_f64(const double* s, int N, const double* Xrt, int64_t ldx, int C,
                                      const double* Yrt, int64_t ldy, int P, int n_grid, double lo, double hi,
                                      int refine, int reml, double* log_delta, int32_t* grid_idx, void* work,
                                      size_t work_bytes, void* stream) {
    FLMM_REQUIRE(s && Xrt && Yrt && log_delta && grid_idx && work && N > C && ldx >= N && ldy >= N && P >= 0 &&
                     n_grid > 0,
                 "flmm_fit_delta_gls_f64: bad arguments");
    int rc = check_c(C, "flmm_fit_delta_gls_f64");
    if (rc) return rc;
    GridWs ws = carve_grid(work, N, C, P, n_grid);
    if (work_bytes < ws.bytes)
        return fail(FLMM_ERR_WORKSPACE, "flmm_fit_delta_gls_f64: need %zu bytes, got %zu", ws.bytes, work_bytes);
    if (P == 0) return FLMM_OK;
    cudaStream_t st = as_stream(stream);
    if ((rc = flmm_delta_grid_nodes(lo, hi, n_grid, ws.grid, stream))) return rc;
    k_gls_grid_prep<<<n_grid, 256, 0, st>>>(s, N, Xrt, ldx, C, ws.grid, ws.W, ws.sum_log, ws.Lg, ws.logdet, ws.bad);
    if ((rc = check_launch("k_gls_grid_prep"))) return rc;
    dim3 g2(ceil_div(P, kEvalWarps), n_grid);
    k_gls_grid_loss<<<g2, 32 * kEvalWarps, 0, st>>>(ws.W, Xrt, ldx, C, Yrt, ldy, N, P, ws.sum_log, ws.Lg, ws.logdet,
                                                     ws.bad, reml, ws.loss);
    if ((rc = check_launch("k_gls_grid_loss"))) return rc;
    k_gls_argmin<<<ceil_div(P, 256), 256, 0, st>>>(ws.loss, n_grid, P, grid_idx);
    if ((rc = check_launch("k_gls_argmin"))) return rc;
    const size_t block_smem = golden_block_smem(N, C);
    if (refine && block_smem <= kBlockSmemMax) {
        // (one bound whatever N: another host thread's call must not lower it under this launch)
        FLMM_CUDA(cudaFuncSetAttribute(k_gls_golden_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlockSmemMax));
        k_gls_golden_block<<<2 * P, kBlockThreads, block_smem, st>>>(s, N, Xrt, ldx, C, Yrt, ldy, ws.grid, n_grid, grid_idx,
                                                                 reml, lo, hi, log_delta);
        return check_launch("k_gls_golden_block");
    }
    const size_t smem = eval_smem_bytes(C);
    FLMM_CUDA(cudaFuncSetAttribute(k_gls_golden, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)eval_smem_bytes(kMaxGlsC)));
    k_gls_golden<<<ceil_div(P, kEvalWarps), 32 * kEvalWarps, smem, st>>>(s, N, Xrt, ldx, C, Yrt, ldy, P, ws.grid,
                                                                          n_grid, grid_idx, refine, reml, lo, hi,
                                                                          log_delta);
    return check_launch("k_gls_golden");
}

extern "C" int flmm_wald_gls_workspace_bytes(int N, int C, int P, size_t* bytes) {
    FLMM_REQUIRE(bytes && N > 0 && C > 0 && P >= 0, "flmm_wald_gls_workspace_bytes: bad arguments");
    *bytes = wald_ws(N, C, P);
    return FLMM_OK;
}

extern "C" int flmm_wald_gls_f64(const double* s, int N, const double* Xrt, int64_t ldx, int C, const double* Yrt,
                                 int64_t ldy, const double* log_delta, int P, int n_real, const double* Srt,
                                 int64_t lds, int M, const int64_t* rows, double* f, double* beta, double* se,
                                 double* sfve, int64_t ldo, double* max_F, void* work, size_t work_bytes,
                                 void* stream) {
    FLMM_REQUIRE(s && Xrt && Yrt && log_delta && max_F && work && N > C + 1 && ldx >= N && ldy >= N && lds >= N &&
                     P >= 0 && M >= 0 && n_real >= 0 && n_real <= P,
                 "flmm_wald_gls_f64: bad arguments");
    FLMM_REQUIRE(n_real == 0 || M == 0 || (rows && f && beta && se && sfve && ldo >= n_real),
                 "flmm_wald_gls_f64: real-column outputs missing");
    FLMM_REQUIRE(M == 0 || Srt, "flmm_wald_gls_f64: Srt is NULL");
    int rc = check_c(C, "flmm_wald_gls_f64");
    if (rc) return rc;
    if (work_bytes < wald_least(N, C, P))
        return fail(FLMM_ERR_WORKSPACE, "flmm_wald_gls_f64: need %zu bytes, got %zu", wald_least(N, C, P), work_bytes);
    if (P == 0 || M == 0) return FLMM_OK;
    cudaStream_t st = as_stream(stream);
    const size_t smem_prep = sizeof(double) * ((kPrepThreads / 32) * static_cast<size_t>(C + 1) * (C + 1) +
                                               static_cast<size_t>(C) * C + (C + 1));
    // Large scans: the products (w o r)^T s, w^T (s o s) and (L^-1 X~^T W) s on the tensor cores from digit planes.  The
    // tile kernel reads two shared-memory operands per FP64 multiply-add and reached 0.87 TFLOP/s (660 columns x 4,000
    // variants x 800 samples, C = 5: 33.9 ms).
    const WaldWs w = carve_wald(work, N, C, P, M, work_bytes);
    if (w.tensor) {
        // (the rotated intercept is one entry, where every centred variant is ~0 and w largest: balanced, it no longer
        // sets its rows' resolution)
        if ((rc = oz_balance(Srt, lds, M, N, w.bal, st))) return rc;
        for (int p0 = 0; p0 < P; p0 += w.pc) {
            const int pc = P - p0 < w.pc ? P - p0 : w.pc;
            const int nr = n_real > p0 ? (n_real - p0 < pc ? n_real - p0 : pc) : 0;
            const int64_t half = static_cast<int64_t>(pc) * N, gs = static_cast<int64_t>(pc) * (M < w.mc ? M : w.mc);
            k_gls_wald_prep<<<pc, kPrepThreads, smem_prep, st>>>(
                s, N, Xrt, ldx, C, Yrt + static_cast<int64_t>(p0) * ldy, ldy, log_delta + p0, 1, w.RW, w.RW + half, N,
                w.Q, static_cast<int64_t>(C) * N, nullptr, w.rWr);
            if ((rc = check_launch("k_gls_wald_prep"))) return rc;
            const OzOperand rw = oz_carve(w.rw_op, pc, N, 2, kOzRowsA), qo = oz_carve(w.q_op, pc * C, N, 1, kOzRowsA);
            if ((rc = oz_digits(rw, 0, w.RW, N, false, w.bal, 1, st))) return rc;
            if ((rc = oz_digits(rw, 1, w.RW + half, N, false, w.bal, 2, st))) return rc;
            // (L^-1 X~^T W W^-1/2 has orthonormal rows: a term is at most sqrt(w^T (s o s)), so its rows are held against w)
            if ((rc = oz_digits(qo, 0, w.Q, N, false, w.bal, 1, st, OzWeights{&rw, C}))) return rc;
            auto out = [&](double* x) { return nr > 0 ? x + p0 : nullptr; };
            for (int m0 = 0; m0 < M; m0 += w.mc) {
                const int mc = M - m0 < w.mc ? M - m0 : w.mc;
                const double* S = Srt + m0 * lds;
                const OzOperand so = oz_carve(w.s_op, mc, N, 2, kOzRowsB);
                if ((rc = oz_digits(so, 0, S, lds, false, w.bal, -1, st))) return rc;
                if ((rc = oz_digits(so, 1, S, lds, true, w.bal, -2, st))) return rc;
                const OzProduct g{w.RW, N, half, S, lds, {false, true}, OzGate::kBalanced, w.G, mc, gs, nullptr, 0};
                const OzProduct gq{w.Q, N, 0, S, lds, {false, false}, OzGate::kTerms, w.Gq, mc, 0, nullptr, 0};
                if ((rc = oz_gemm(rw, so, g, st))) return rc;
                if ((rc = oz_gemm(qo, so, gq, st))) return rc;
                if ((rc = wald_finish(w.G, w.G + gs, w.Gq, C, mc, w.rWr, static_cast<double>(N - C - 1), pc, nr, mc,
                                      nr > 0 ? rows + m0 : nullptr, out(f), out(beta), out(se), out(sfve), ldo,
                                      max_F + p0, st)))
                    return rc;
            }
        }
        return FLMM_OK;
    }
    const size_t smem_wald = sizeof(double) * (static_cast<size_t>(WP) * (C + 2) * WK + WM * WK);
    for (int q0 = 0; q0 < P; q0 += w.pc) {
        const int pc = P - q0 < w.pc ? P - q0 : w.pc;
        double* Lv = static_cast<double*>(work);
        double* Lp = Lv + static_cast<size_t>(pc) * (C + 2) * N;
        double* rWr = Lp + static_cast<size_t>(pc) * C * C;
        k_gls_wald_prep<<<pc, kPrepThreads, smem_prep, st>>>(
            s, N, Xrt, ldx, C, Yrt + static_cast<int64_t>(q0) * ldy, ldy, log_delta + q0, 0, Lv,
            Lv + static_cast<int64_t>(C + 1) * N, static_cast<int64_t>(C + 2) * N, Lv + N,
            static_cast<int64_t>(C + 2) * N, Lp, rWr);
        if ((rc = check_launch("k_gls_wald_prep"))) return rc;
        const int nr = n_real - q0 > 0 ? (n_real - q0 < pc ? n_real - q0 : pc) : 0;
        dim3 grid(ceil_div(M, WM), ceil_div(pc, WP));
        // detail outputs exist (and are offset) only for chunks holding real columns
        double* fo = nr > 0 ? f + q0 : nullptr;
        double* bo = nr > 0 ? beta + q0 : nullptr;
        double* so = nr > 0 ? se + q0 : nullptr;
        double* vo = nr > 0 ? sfve + q0 : nullptr;
        auto launch = [&](auto kernel) {
            kernel<<<grid, WT, smem_wald, st>>>(Lv, Lp, rWr, N, C, pc, nr, Srt, lds, M, rows, fo, bo, so, vo, ldo,
                                                max_F + q0);
        };
        if (C + 2 <= 8) launch(k_gls_wald<8>);
        else if (C + 2 <= 16) launch(k_gls_wald<16>);
        else launch(k_gls_wald<32>);
        if ((rc = check_launch("k_gls_wald"))) return rc;
    }
    return FLMM_OK;
}

extern "C" int flmm_shift_diagonal_f64(double* A, int N, int64_t lda, double value, void* stream) {
    FLMM_REQUIRE(A && N > 0 && lda >= N, "flmm_shift_diagonal_f64: bad arguments");
    k_shift_diagonal<<<ceil_div(N, 256), 256, 0, as_stream(stream)>>>(A, N, lda, value);
    return check_launch("k_shift_diagonal");
}

extern "C" int flmm_clamp_nonneg_f64(const double* x, int64_t n, double* y, void* stream) {
    FLMM_REQUIRE((x && y) || n == 0, "flmm_clamp_nonneg_f64: bad arguments");
    if (n == 0) return FLMM_OK;
    k_clamp_nonneg<<<ceil_div(n, 256), 256, 0, as_stream(stream)>>>(x, n, y);
    return check_launch("k_clamp_nonneg");
}
