// Plain FP64 form of the null-model delta fit (fasterlmm/core.py:525-595): the (G, P) grid of ML -2 log L, its
// first argmin per column, and the reference's 50-step golden-section refinement on [grid[i-1], grid[i+1]].
//
// The loss is evaluated with the reference's operation order, and every a + k * (b - a) bracket update uses
// non-contracting FP64 intrinsics, so each step rounds like the reference's separate tensor operations.  Summation
// order over the eigenvalues differs (warp / tile sums), which is why the refined value agrees with the reference
// to its own FP64 noise rather than bit for bit.
#include <math.h>

#include "flmm_common.cuh"

using namespace flmm;

namespace {

constexpr double kLog2Pi = 1.8378770664093453;  // log(2 pi) in FP64, the reference's log2pi constant

// The low-rank model (fasterlmm/lowrank.py:131-151) adds, per column, the off-rank quadratic form yy_off / delta
// and (Neff - k) log delta to the log determinant, and its Neff is N - D rather than the spectrum length k.  The
// compat fit is the special case yy = NULL, n_logd = 0, neff = k.
struct OffRank {
    const double* yy;  // (P,) off-rank residual sum of squares, or NULL
    double neff;       // sample count of the variance estimate
    double n_logd;     // count of extra log(delta) terms in log det V
};

// ML -2 log L from the weighted sum yWy and log det V (fasterlmm/core.py:538-542, fasterlmm/lowrank.py:144-151)
__device__ __forceinline__ double ml_loss(double yWy, double sum_log_sd, double delta, double yy_off,
                                          const OffRank& o) {
    double rWr = fmax(o.yy ? add_rn(yWy, yy_off / delta) : yWy, kPosFloor);
    double sigma2 = rWr / o.neff;
    double t = add_rn(add_rn(kLog2Pi, log(sigma2)), 1.0);
    const double logdet = o.n_logd != 0.0 ? add_rn(sum_log_sd, mul_rn(o.n_logd, log(delta))) : sum_log_sd;
    return add_rn(mul_rn(o.neff, t), logdet);
}

// Wg[g, n] = 1 / (s[n] + exp(grid[g])), sum_log[g] = sum_n log(s[n] + exp(grid[g])); one block per grid node
__global__ void k_grid_weights(const double* __restrict__ s, int Neff, const double* __restrict__ grid,
                               double* __restrict__ Wg, double* __restrict__ sum_log) {
    __shared__ double red[32];
    const int g = blockIdx.x;
    const double delta = exp(grid[g]);
    double acc = 0.0;
    for (int n = threadIdx.x; n < Neff; n += blockDim.x) {
        double sd = s[n] + delta;
        Wg[static_cast<int64_t>(g) * Neff + n] = 1.0 / sd;
        acc += log(sd);
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) sum_log[g] = v;
    }
}

// Grid loss and first argmin over g for a tile of 16 RP columns; g is walked in tiles of 64.  yWy[g, p] =
// sum_n Wg[g, n] UY[p, n]^2 is the (G x Neff) x (Neff x P) product of fasterlmm/core.py:537, one chain of multiply-adds
// over n per (g, p) whatever the tile.  The FP64 pipe is the bound, so tiles of 16 columns (RP = 1) are as good as tiles
// of 64 and give four times the blocks: 2,100 columns are 33 blocks of 64 on 152 SMs.
constexpr int TG = 64, TK = 16, NT = 256;

template <int RP>
__global__ void __launch_bounds__(NT)
k_grid_argmin(const double* __restrict__ Wg, const double* __restrict__ sum_log, const double* __restrict__ grid,
              const double* __restrict__ UYt, int64_t ldu, int Neff, int P, int G, OffRank off,
              int32_t* __restrict__ idx_out) {
    constexpr int TP = 16 * RP;
    __shared__ double Ws[TK][TG + 1];
    __shared__ double Us[TK][TP + 1];
    __shared__ double red_v[16][TP];
    __shared__ int red_i[16][TP];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int p0 = blockIdx.x * TP;
    double best = INFINITY;
    int best_g = 0;
    for (int g0 = 0; g0 < G; g0 += TG) {
        double acc[4][RP] = {};
        for (int k0 = 0; k0 < Neff; k0 += TK) {
#pragma unroll
            for (int l = 0; l < (TG * TK) / NT; ++l) {
                int t = tid + l * NT, g = t / TK, k = t % TK;
                int gg = g0 + g, gk = k0 + k;
                Ws[k][g] = (gg < G && gk < Neff) ? Wg[static_cast<int64_t>(gg) * Neff + gk] : 0.0;
            }
#pragma unroll
            for (int l = 0; l < (TP * TK) / NT; ++l) {
                int t = tid + l * NT, p = t / TK, k = t % TK;
                int gp = p0 + p, gk = k0 + k;
                double u = (gp < P && gk < Neff) ? UYt[static_cast<int64_t>(gp) * ldu + gk] : 0.0;
                Us[k][p] = u * u;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < TK; ++k) {
                double a[4], b[RP];
#pragma unroll
                for (int r = 0; r < 4; ++r) a[r] = Ws[k][ty + 16 * r];
#pragma unroll
                for (int c = 0; c < RP; ++c) b[c] = Us[k][tx + 16 * c];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < RP; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
            }
            __syncthreads();
        }
        // this thread's nodes are g0 + ty + 16 r, ascending in r: keep the first minimum per column
#pragma unroll
        for (int c = 0; c < RP; ++c) {
            double bv = INFINITY;
            int bi = G;
            const int pc = p0 + tx + 16 * c;
            const double yy = (off.yy && pc < P) ? off.yy[pc] : 0.0;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                int g = g0 + ty + 16 * r;
                if (g < G) {
                    const double dg = (off.yy || off.n_logd != 0.0) ? exp(grid[g]) : 1.0;  // compat needs no delta
                    double v = ml_loss(acc[r][c], sum_log[g], dg, yy, off);
                    if (v < bv) { bv = v; bi = g; }
                }
            }
            red_v[ty][tx + 16 * c] = bv;
            red_i[ty][tx + 16 * c] = bi;
        }
        __syncthreads();
        if (tid < TP) {
            for (int r = 0; r < 16; ++r) {
                double v = red_v[r][tid];
                int gi = red_i[r][tid];
                if (v < best || (v == best && gi < best_g)) { best = v; best_g = gi; }
            }
        }
        __syncthreads();
    }
    if (tid < TP && p0 + tid < P) idx_out[p0 + tid] = best_g;
}

// log_delta[p] = grid[idx[p]]: the fit without refinement
__global__ void k_grid_pick(const double* __restrict__ grid, const int32_t* __restrict__ idx, int P,
                            double* __restrict__ log_delta) {
    const int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (p < P) log_delta[p] = grid[idx[p]];
}

// Golden-section search (fasterlmm/core.py:545-558, :577-595), 50 steps that each compare two losses.  Its value is the
// list of those comparisons: the last third of them compare rounding noise, so every loss that decides one has to keep its
// bits (k_golden), but the first half compare losses that are far apart, and those need only be good enough to be sure of
// the sign (k_golden_certain).  The list is handed over in the output word: bit k is step k's answer, the top byte how many
// steps are decided.
constexpr int kGoldenSteps = 50;

__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The steps whose answer is certain, one warp per column.  The sums come from groups of up to 16 eigenvalues as one
// fraction and one logarithm, sum u^2 / x = num / den and sum log x = log den, ~7 operations of the FP64 pipe an eigenvalue
// for the ~60 of a division and a logarithm each, and the point that a step shares with the one before is not evaluated
// again.  A step is certain when the two losses differ by more than twice what rounding can make of them here and in
// k_golden together.  exp and log are taken to be within one unit in the last place (CUDA's documented bounds; the same
// delta goes into both sides).  With u = 2^-53 and n eigenvalues, to first order and both sides: sum u^2 / x is a sum of positive
// terms, relative error below (n / 30 + 58) u; sum log x is off by at most (n / 30 + 20) u sum |log x| + n u; a shared
// point whose position differs in its last bits moves the loss by at most (neff + n + |n_logd|) times that.  The first step
// that is not certain ends the list, as does anything out of the range of these bounds.
// 2,100 columns x 596 eigenvalues: 22 of the 50 steps on average, the whole fit 10.5 -> 7.0 ms.
constexpr int kCertainWarps = 4, kGroup = 16;

__global__ void __launch_bounds__(32 * kCertainWarps)
k_golden_certain(const double* __restrict__ s, int Neff, const double* __restrict__ UYt, int64_t ldu, int P,
                 const double* __restrict__ grid, int G, const int32_t* __restrict__ idx, OffRank off,
                 double* __restrict__ list) {
    const int lane = threadIdx.x & 31;
    const int64_t p = static_cast<int64_t>(blockIdx.x) * kCertainWarps + (threadIdx.x >> 5);
    if (p >= P) return;
    const double* u = UYt + p * ldu;
    const double yy = off.yy ? off.yy[p] : 0.0;
    Bracket br(grid, G, idx[p]);
    double smin = INFINITY, smax = -INFINITY;
    for (int n = lane; n < Neff; n += 32) {
        smin = fmin(smin, s[n]);
        smax = fmax(smax, s[n]);
    }
    const double xlo = -warp_max(-smin) + exp(br.a), xhi = warp_max(smax) + exp(br.b);
    const double edge = fmax(fmax(fabs(br.a), fabs(br.b)), 1.0);
    const double rnd = 0x1p-53, n = Neff, nd = fabs(off.n_logd);
    // what does not depend on the loss: the logarithms' share, and that of the extra log(delta)
    const double labs = n * fmax(fabs(log(xlo)), fabs(log(xhi)));
    const double fixed = labs * (n / 30.0 + 26.0) + n + 12.0 * nd * edge;
    bool certain = xlo > 0x1p-50 && xhi < 0x1p50 && yy >= 0.0;

    double bound = 0.0;  // of the loss of the latest call
    auto loss_at = [&](double x) {
        const double delta = exp(x);
        double q = 0.0, l = 0.0;
        for (int n0 = 0; n0 < Neff; n0 += 32 * kGroup) {
            double num = 0.0, den = 1.0;
            // pairs of eigenvalues, joined one after another
#pragma unroll
            for (int j = 0; j < kGroup; j += 2) {
                if (n0 + 32 * j >= Neff) break;
                const int i0 = n0 + 32 * j + lane, i1 = i0 + 32;
                double x0 = 1.0, x1 = 1.0, u0 = 0.0, u1 = 0.0;
                if (i0 < Neff) {
                    x0 = s[i0] + delta;
                    u0 = u[i0];
                }
                if (i1 < Neff) {
                    x1 = s[i1] + delta;
                    u1 = u[i1];
                }
                const double pn = fma(u0 * u0, x1, u1 * u1 * x0), pd = x0 * x1;
                num = fma(num, pd, pn * den);
                den *= pd;
            }
            q += num / den;
            l += log(den);
        }
        q = warp_sum(q);
        l = warp_sum(l);
        if (off.yy) q += yy / delta;
        certain = certain && q > 0x1p-200 && q < 0x1p300;
        const double ls = log(fmax(q, kPosFloor) / off.neff);
        bound = rnd * (off.neff * (n / 30.0 + 90.0 + 10.0 * fabs(ls)) + fixed);
        return off.neff * (kLog2Pi + ls + 1.0) + l + off.n_logd * x;
    };

    unsigned long long bits = 0;
    int it = 0;
    double xc = br.c(), xd = br.d();
    double fc = loss_at(xc), bc = bound, fd = loss_at(xd), bd = bound;
    while (certain && it < kGoldenSteps) {
        const double slope = off.neff + n + nd;
        const double tol = 2.0 * (bc + bd + slope * (fabs(xc - br.c()) + fabs(xd - br.d()) + 16.0 * rnd));
        const bool left = fd - fc > tol;
        if (!left && !(fc - fd > tol)) break;
        if (left) bits |= 1ull << it;
        ++it;
        br.narrow(left);
        if (it == kGoldenSteps) break;
        if (left) {
            xd = xc, fd = fc, bd = bc;
            xc = br.c(), fc = loss_at(xc), bc = bound;
        } else {
            xc = xd, fc = fd, bc = bd;
            xd = br.d(), fd = loss_at(xd), bd = bound;
        }
    }
    if (lane == 0) list[p] = __longlong_as_double(static_cast<long long>(bits | static_cast<unsigned long long>(it) << 56));
}

// The other steps, one block per column.  The terms of a step's two evaluations, a division and a logarithm per eigenvalue,
// are formed by all threads into shared memory, kTermChunk eigenvalues at a time; one warp per sum then adds them, lane l
// the terms l, l + 32, ... in order and the lanes by a butterfly.  A point that is, to the bit, one of the step before keeps
// its loss (one step in five has one).  The search stops at the rounding noise of the loss, so
// this order is part of the result.  Bound by the FP64 pipe (~60 operations a term); a warp per column had few columns wait
// for 2 Neff / 32 terms one after another on few SMs: all steps of 176 columns x 450 eigenvalues 5.6 -> 1.8 ms, 220 x 880
// 8.7 -> 2.8 ms, 2,100 x 596 12.7 -> 11.0 ms.
constexpr int kBlockThreads = 256, kTermChunk = 1024;

__global__ void __launch_bounds__(kBlockThreads)
k_golden(const double* __restrict__ s, int Neff, const double* __restrict__ UYt, int64_t ldu,
         const double* __restrict__ grid, int G, const int32_t* __restrict__ idx, double lo, double hi, OffRank off,
         double* __restrict__ log_delta) {
    __shared__ double term[2][2][kTermChunk];  // [evaluation][w u u, log]
    __shared__ double delta_s[2], sum_s[2][2], loss_s[2];
    __shared__ int kept_s[2];
    const int64_t p = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* u = UYt + p * ldu;
    const double yy = off.yy ? off.yy[p] : 0.0;
    const unsigned long long list = static_cast<unsigned long long>(__double_as_longlong(log_delta[p]));
    const int done = static_cast<int>(list >> 56);
    __syncthreads();  // every thread has read the list; thread 0 overwrites it
    // threads 0 and 32 carry the search, one evaluation each
    const bool lead = tid == 0 || tid == 32;
    const int my_e = tid >> 5;
    Bracket br(grid, G, idx[p]);
    if (lead)
        for (int it = 0; it < done; ++it) br.narrow(list >> it & 1);
    for (int it = done; it < kGoldenSteps; ++it) {
        double delta = 0.0, kept_loss = 0.0;
        bool kept = false;
        if (lead) {
            kept = it > done && br.narrow_kept(loss_s, my_e, &kept_loss);
            delta = exp(my_e ? br.d() : br.c());
            delta_s[my_e] = delta;
            kept_s[my_e] = kept;
        }
        __syncthreads();
        // evaluations e0 .. e1
        const int e0 = kept_s[0], e1 = 2 - kept_s[1];
        double acc = 0.0;  // warps 0..3: sum (warp & 1) of evaluation warp >> 1
        const bool sums = warp < 4 && (warp >> 1) >= e0 && (warp >> 1) < e1;
        for (int n0 = 0; n0 < Neff; n0 += kTermChunk) {
            const int m = min(kTermChunk, Neff - n0);
            for (int t = e0 * m + tid; t < e1 * m; t += kBlockThreads) {
                const int e = t >= m, n = t - (e ? m : 0);
                const double sd = s[n0 + n] + delta_s[e];
                const double w = 1.0 / sd;
                const double un = u[n0 + n];
                term[e][0][n] = mul_rn(mul_rn(w, un), un);
                term[e][1][n] = log(sd);
            }
            __syncthreads();
            if (sums) {
                const double* x = term[warp >> 1][warp & 1];
                for (int n = lane; n < m; n += 32) acc += x[n];
            }
            __syncthreads();
        }
        if (sums) {
            acc = warp_sum(acc);
            if (lane == 0) sum_s[warp >> 1][warp & 1] = acc;
        }
        __syncthreads();
        if (lead) loss_s[my_e] = kept ? kept_loss : ml_loss(sum_s[my_e][0], sum_s[my_e][1], delta, yy, off);
        __syncthreads();
    }
    if (tid == 0) {
        if (done < kGoldenSteps) br.narrow(loss_s[0] < loss_s[1]);
        log_delta[p] = fmin(fmax(mul_rn(0.5, add_rn(br.a, br.b)), lo), hi);
    }
}

size_t fit_ws(int Neff, int G) {
    return sizeof(double) * (static_cast<size_t>(G) * Neff + 2 * static_cast<size_t>(G)) + 256;
}

}  // namespace

extern "C" int flmm_fit_delta_f64_workspace_bytes(int Neff, int n_grid, size_t* bytes) {
    FLMM_REQUIRE(bytes && Neff > 0 && n_grid > 0, "flmm_fit_delta_f64_workspace_bytes: bad arguments");
    *bytes = fit_ws(Neff, n_grid);
    return FLMM_OK;
}

namespace {

int fit_delta_impl(const double* s, int Neff, const double* UYt, int64_t ldu, int P, int n_grid, double lo, double hi,
                   int refine, const OffRank& off, double* log_delta, int32_t* grid_idx, void* work, size_t work_bytes,
                   void* stream, const char* fn) {
    if (work_bytes < fit_ws(Neff, n_grid))
        return fail(FLMM_ERR_WORKSPACE, "%s: need %zu bytes, got %zu", fn, fit_ws(Neff, n_grid), work_bytes);
    if (P == 0) return FLMM_OK;
    cudaStream_t st = as_stream(stream);
    double* Wg = static_cast<double*>(work);
    double* sum_log = Wg + static_cast<size_t>(n_grid) * Neff;
    double* grid = sum_log + n_grid;
    int rc = flmm_delta_grid_nodes(lo, hi, n_grid, grid, stream);
    if (rc) return rc;
    k_grid_weights<<<n_grid, 256, 0, st>>>(s, Neff, grid, Wg, sum_log);
    if ((rc = check_launch("k_grid_weights"))) return rc;
    int sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    if (P >= 64 * sms)
        k_grid_argmin<4><<<ceil_div(P, 64), NT, 0, st>>>(Wg, sum_log, grid, UYt, ldu, Neff, P, n_grid, off, grid_idx);
    else
        k_grid_argmin<1><<<ceil_div(P, 16), NT, 0, st>>>(Wg, sum_log, grid, UYt, ldu, Neff, P, n_grid, off, grid_idx);
    if ((rc = check_launch("k_grid_argmin"))) return rc;
    if (refine) {
        if (refine == FLMM_REFINE_EVERY_STEP) {
            FLMM_CUDA(cudaMemsetAsync(log_delta, 0, sizeof(double) * P, st));  // empty lists
        } else {
            k_golden_certain<<<ceil_div(P, kCertainWarps), 32 * kCertainWarps, 0, st>>>(s, Neff, UYt, ldu, P, grid, n_grid,
                                                                                       grid_idx, off, log_delta);
            if ((rc = check_launch("k_golden_certain"))) return rc;
        }
        k_golden<<<P, kBlockThreads, 0, st>>>(s, Neff, UYt, ldu, grid, n_grid, grid_idx, lo, hi, off, log_delta);
        return check_launch("k_golden");
    }
    k_grid_pick<<<ceil_div(P, 256), 256, 0, st>>>(grid, grid_idx, P, log_delta);
    return check_launch("k_grid_pick");
}

}  // namespace

extern "C" int flmm_fit_delta_f64(const double* s, int Neff, const double* UYt, int64_t ldu, int P, int n_grid,
                                  double lo, double hi, int refine, double* log_delta, int32_t* grid_idx, void* work,
                                  size_t work_bytes, void* stream) {
    FLMM_REQUIRE(s && UYt && log_delta && grid_idx && work && Neff > 0 && n_grid > 0 && ldu >= Neff && P >= 0,
                 "flmm_fit_delta_f64: bad arguments");
    const OffRank off{nullptr, static_cast<double>(Neff), 0.0};
    return fit_delta_impl(s, Neff, UYt, ldu, P, n_grid, lo, hi, refine, off, log_delta, grid_idx, work, work_bytes,
                          stream, "flmm_fit_delta_f64");
}

extern "C" int flmm_fit_delta_lowrank_f64(const double* s, int k, const double* UYt, int64_t ldu, const double* yy_off,
                                          int Neff, int P, int n_grid, double lo, double hi, int refine,
                                          double* log_delta, int32_t* grid_idx, void* work, size_t work_bytes,
                                          void* stream) {
    FLMM_REQUIRE(s && UYt && yy_off && log_delta && grid_idx && work && k > 0 && Neff > 0 && n_grid > 0 && ldu >= k &&
                     P >= 0,
                 "flmm_fit_delta_lowrank_f64: bad arguments");
    // Neff - k may be negative: with k >= N the reference's basis can keep O(1e-17) directions of the projected-out
    // space, each adding log(s + delta) ~ log(delta), which the negative count cancels (fasterlmm/lowrank.py:88-94)
    const OffRank off{yy_off, static_cast<double>(Neff), static_cast<double>(Neff - k)};
    return fit_delta_impl(s, k, UYt, ldu, P, n_grid, lo, hi, refine, off, log_delta, grid_idx, work, work_bytes,
                          stream, "flmm_fit_delta_lowrank_f64");
}
