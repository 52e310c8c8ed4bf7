// Batched FP32 symmetric eigendecomposition of the projected LOCO kinships (N below 2,500), the fast form's
// replacement for the library's batched eigensolver.  The reference decomposes each kinship in FP64
// (fasterlmm/core.py:54-77, torch.linalg.eigh); the fast form takes an FP32 decomposition and refines it
// (flmm_eigh_refine_f32), so only FP32-quality eigenpairs are needed here.
//
// Five stages, all matrices of the batch side by side:
//
// 1. k_sytrd_cluster: Householder tridiagonalisation A = Q T Q^T, one thread-block cluster of 2 to 16 CTAs per
//    matrix (one CTA per SM).  The FP32 matrix stays in global memory (L2-resident for the batch sizes used), rows
//    dealt round-robin to the cluster's CTAs.  Column k's reflector is formed redundantly by every CTA, each CTA
//    computes p = tau W v for its rows and stores it into every CTA's shared memory (distributed shared memory), so
//    after the barrier each CTA reads only its own.  The symmetric rank-2 update W -= v w^T + w v^T is applied lazily,
//    in the passes that form the next columns' W v, and a row is written back with every second update only; the next
//    pivot row gets what is pending in registers in every CTA, which forms the next reflector from it.  Both products
//    of an update term are rounded before the add, so W stays exactly symmetric.  One cluster barrier per column.
//    What bounds it: the write path to L2 (88% of its cycles with a write per column; two updates in a row cost less than
//    a write), then the chain of a column: barrier, p^T v, w, reflector, whose loads pass during the row pass.  20 x 1,000
//    11.3 -> 8.2 ms, 8 x 1,600 21.7 -> 16.3, 22 x 563 3.46 -> 2.48.  Keeping rows in shared memory (all of them at 563),
//    and smaller blocks of loads ahead of the one at work, gave nothing or less.
// 2. k_tridiag_bisect: each eigenvalue of T by multisection on FP32 Sturm counts (ascending, by index; three points
//    per step, so 24 steps narrow the bracket as 48 halvings would).
// 3. k_tridiag_invit: each eigenvector of T by inverse iteration in FP64 (LDL^T of T - lambda I with a pivot floor,
//    three solves from a fixed pseudo-random start, the first fused with the factorisation), one thread each.
// 4. k_cluster_orth: eigenvalues closer than kClusterTol * ||T|| form a cluster; one block orthonormalises its
//    vectors (modified Gram-Schmidt in FP64).  Each vector of a cluster has converged into the cluster's invariant
//    subspace from its own start, so the result is an orthonormal basis of that subspace.
// 5. k_wy_factors + k_backtransform: the reflectors in blocks of kWy as I - V T V^T (forward, columnwise), applied to
//    column tiles of the eigenvector matrix of T held in shared memory, last block first; the result is written as
//    one eigenvector per row.
//
// Every loop is bounded by N and fixed iteration counts; the only waits are cluster barriers that every CTA of the
// cluster reaches on the same trip count.
#include <math.h>

#include <algorithm>
#include <mutex>
#include <stdint.h>

#include "flmm_common.cuh"

using namespace flmm;

namespace {

constexpr int kMaxClusterCtas = 16;  // beyond 8 the size is not portable
constexpr int kMaxParts = 8;         // partial sums of p^T v
constexpr int kSytrdThreads = 512;
// a column's cycles on average: its row pass at N = 1,000 in one CTA, what every CTA repeats, and the barrier's share per CTA
constexpr double kRowPassCycles = 75e3, kColumnCycles = 3e3, kCtaCycles = 50;
constexpr int kPend = 2;           // column updates that gather before the rows are written
constexpr int kRowsPerWarp = 4;    // rows a warp of the tridiagonalisation works on at once
constexpr int kDotRows = 4;        // rows of p^T v that follow one another in a chain (part of the result)
constexpr int kOwnCols = 5;        // columns of a thread in the vector passes: N <= 512 * 5
constexpr int kLoadsPerRow = 8;    // loads of each of them a lane has in flight
constexpr int kWy = 16;            // reflectors per WY block
constexpr int kChunk = 64;         // rows of two V blocks staged at a time in the back-transform
constexpr int kRing = 3;           // such chunks in shared memory: one read by each phase, one on its way
static_assert(kWy == 16 && kChunk == 64, "the back-transform's thread layout");
// the FP32 shift is within ~1e-7 ||T|| of its eigenvalue: at the cluster cut (a gap of 1e-5 ||T||) each solve shrinks
// the neighbour by ~1e-2, so three solves leave ~1e-6 of it (two left pairs near the cut ~1e-4 from orthogonal)
constexpr int kInvitSolves = 3;
constexpr int kInvitBlock = 16;     // elements whose loads a recurrence pass issues ahead
constexpr double kClusterTol = 1e-5;
constexpr int kSectPts = 3;        // points per multisection step of the eigenvalue brackets (its quarters)
constexpr int kBisectSteps = 24;   // 4^-24 = 2^-48 of the Gershgorin interval
// one warp a block: the eigenvalues' warps spread over all SMs (20 x 1,000 with blocks of 128: 0.67 -> 0.60 and, inverse
// iteration, 2.32 -> 2.02 ms; 8 x 1,600 0.88 -> 0.74 and 2.95 -> 2.90)
constexpr int kBisectThreads = 32, kInvitThreads = 32;

__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_index() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// FP32 store into the shared memory of the cluster's CTA `rank` at the address of `p` in this CTA (made visible to it
// by the next cluster barrier)
__device__ __forceinline__ void st_remote(float* p, uint32_t rank, float v) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// block-wide FP32 sum (all threads get it); red holds >= 32 floats
__device__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    float t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0f;
    if (wid == 0) t = warp_sum(t);
    if (threadIdx.x == 0) red[0] = t;
    __syncthreads();
    return red[0];
}

// W (batch, N, N) FP32 symmetric, full storage, overwritten: row k holds the reflector v_k on columns k+1..N-1
// (v_k[k+1] = 1).  d (batch, N), e (batch, N), tau (batch, N): T's diagonal, off-diagonal (e[k] = T[k][k+1]) and the
// reflector scalars (tau[N-2] = tau[N-1] = 0).  The cluster size C is the launch's (%cluster_nctarank); CTA r owns
// the rows i with i % C == r.
//
// Step k: (B) each CTA applies its rows' pending updates (one or two columns; stored if two, but for row k + 1) and forms
// p_i = tau_k W[i, k+1:] v_k; one cluster barrier; (C) every CTA adds up p^T v, forms w_k, applies what is pending and column
// k's update to row k + 1 in registers (as it was last written: loaded before (B), since nobody writes it in this step) and
// forms the next reflector v_{k+1} -- redundantly in every CTA, so no second barrier is needed.
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

struct Reflector {
    float d, beta, tau;
};

// From x = row entries x[k .. N-1] in xs[] (xs[j] for j >= k + 1; d passed in): the reflector of column k into v[]
// (v[k+1] = 1, v[j] = x_j / (alpha - beta) for j >= k + 2), as LAPACK's larfg.  Every thread of the CTA calls it.
__device__ Reflector make_reflector(float d, float alpha, float ss_partial, float* v, int k, int N, float* red) {
    const float sigma = block_sum(ss_partial, red);
    Reflector R{d, alpha, 0.0f};
    float scal = 0.0f;
    if (sigma > 0.0f) {
        R.beta = -copysignf(sqrtf(fmaf(alpha, alpha, sigma)), alpha);
        R.tau = (R.beta - alpha) / R.beta;
        scal = 1.0f / (alpha - R.beta);
    }
    for (int j = k + 2 + threadIdx.x; j < N; j += blockDim.x) v[j] *= scal;
    if (threadIdx.x == 0) v[k + 1] = 1.0f;
    __syncthreads();
    return R;
}

// kQ rows i0, i0 + di, ... (rows of N entries from W on) at columns k + 1 ..: the kM pending updates, oldest first, whose
// vectors start at sm[ov[m]] and sm[ow[m]], stored when kM is kPend (not row k + 1); then p_i = tau row . v into every CTA's
// copy of p.  Every lane adds up its columns k + 1 + lane + 32 t in order.
extern __shared__ float sytrd_sm[];

template <int kM, int kQ>
__device__ __forceinline__ void update_rows(float* W, int N, int k, int i0, int di, int oc, const int (&ov)[kPend],
                                            const int (&ow)[kPend], float tau, int C, float* pb) {
    const int lane = threadIdx.x & 31, len = N - k - 1;
    const bool next = i0 == k + 1;
    float* row0 = W + static_cast<int64_t>(i0) * N + k + 1 + lane;
    const int64_t dr = static_cast<int64_t>(di) * N;
    float vi[kM > 0 ? kM : 1][kQ], wi[kM > 0 ? kM : 1][kQ], acc[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        acc[q] = 0.0f;
#pragma unroll
        for (int m = 0; m < kM; ++m) {
            vi[m][q] = sytrd_sm[ov[m] + i0 + q * di];
            wi[m][q] = sytrd_sm[ow[m] + i0 + q * di];
        }
    }
    const float* v = sytrd_sm + oc + k + 1 + lane;
    float* at[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) at[q] = row0 + q * dr;
    auto take = [&](const float (&x)[kQ], int u) {
        const float vj = v[32 * u];
        float vp[kM > 0 ? kM : 1], wp[kM > 0 ? kM : 1];
#pragma unroll
        for (int m = 0; m < kM; ++m) {
            vp[m] = v[ov[m] - oc + 32 * u];
            wp[m] = v[ow[m] - oc + 32 * u];
        }
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
            float y = x[q];
#pragma unroll
            for (int m = 0; m < kM; ++m) y -= __fmul_rn(vi[m][q], wp[m]) + __fmul_rn(wi[m][q], vp[m]);
            if (kM == kPend && !(q == 0 && next)) at[q][32 * u] = y;
            acc[q] = fmaf(y, vj, acc[q]);
        }
    };
    int rest = len;
#pragma unroll 1
    for (; rest >= 32 * kLoadsPerRow; rest -= 32 * kLoadsPerRow) {
        float x[kLoadsPerRow][kQ];
#pragma unroll
        for (int u = 0; u < kLoadsPerRow; ++u)
#pragma unroll
            for (int q = 0; q < kQ; ++q) x[u][q] = at[q][32 * u];
#pragma unroll
        for (int u = 0; u < kLoadsPerRow; ++u) take(x[u], u);
        v += 32 * kLoadsPerRow;
#pragma unroll
        for (int q = 0; q < kQ; ++q) at[q] += 32 * kLoadsPerRow;
    }
    if (rest > 0) {
        float x[kLoadsPerRow][kQ];
#pragma unroll
        for (int u = 0; u < kLoadsPerRow; ++u)
#pragma unroll
            for (int q = 0; q < kQ; ++q) x[u][q] = 32 * u + lane < rest ? at[q][32 * u] : 0.0f;
#pragma unroll
        for (int u = 0; u < kLoadsPerRow; ++u)
            if (32 * u + lane < rest) take(x[u], u);
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
        const float pi = tau * warp_sum(acc[q]);
        // p_i into every CTA's copy of p (lane l to CTA l): after the barrier all of p is local
        if (lane < C) st_remote(&pb[i0 + q * di], static_cast<uint32_t>(lane), pi);
    }
}

// A warp's rows i0, i0 + di, ..., kRowsPerWarp at a time.
template <int kM>
__device__ __forceinline__ void update_all(float* W, int N, int k, int i0, int di, int oc, const int (&ov)[kPend],
                                           const int (&ow)[kPend], float tau, int C, float* pb) {
    for (; i0 + (kRowsPerWarp - 1) * di < N; i0 += kRowsPerWarp * di)
        update_rows<kM, kRowsPerWarp>(W, N, k, i0, di, oc, ov, ow, tau, C, pb);
    if (i0 + di < N) {
        update_rows<kM, 2>(W, N, k, i0, di, oc, ov, ow, tau, C, pb);
        i0 += 2 * di;
    }
    if (i0 < N) update_rows<kM, 1>(W, N, k, i0, di, oc, ov, ow, tau, C, pb);
}

__global__ void __launch_bounds__(kSytrdThreads, 1)
k_sytrd_cluster(float* __restrict__ W, int N, int parts, float* __restrict__ d_out, float* __restrict__ e_out,
                float* __restrict__ tau_out) {
    float* const sm = sytrd_sm;
    const int Np = (N + 3) & ~3;
    float* const vbuf = sm;                        // v_k in slot k % (kPend + 1)
    float* const wbuf = sm + (kPend + 1) * Np;     // w_k likewise
    float* const pbuf = wbuf + (kPend + 1) * Np;         // p of column k in slot k % 2
    float* red = pbuf + 2 * Np;      // 2 x 32 floats
    float* part = red + 64;          // partial sums of p^T v
    float* scal2 = part + kMaxParts;  // d and alpha of the next reflector
    const int C = static_cast<int>(cluster_size());
    const int b = static_cast<int>(cluster_index());
    const int r = static_cast<int>(cta_rank());
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = kSytrdThreads >> 5;
    float* Wb = W + static_cast<int64_t>(b) * N * N;
    float* db = d_out + static_cast<int64_t>(b) * N;
    float* eb = e_out + static_cast<int64_t>(b) * N;
    float* tb = tau_out + static_cast<int64_t>(b) * N;
    cluster_barrier();          // every CTA runs: its shared memory may be written
    int first = r > 0 ? r : C;  // first row of this CTA past row k
    int first_dot = 1 % parts;  // k + 1 modulo parts
    Reflector R{0.0f, 0.0f, 0.0f};
    if (N >= 3) {  // reflector of column 0 from the untouched row 0
        float ss = 0.0f;
        for (int j = 2 + threadIdx.x; j < N; j += kSytrdThreads) {
            const float x = Wb[j];
            vbuf[j] = x;
            ss = fmaf(x, x, ss);
        }
        R = make_reflector(Wb[0], Wb[1], ss, vbuf, 0, N, red);
    }
    for (int k = 0; k + 2 < N; ++k) {
        const float* vc = vbuf + k % (kPend + 1) * Np;
        float* vn = vbuf + (k + 1) % (kPend + 1) * Np;  // v_{k - kPend}, then v_{k+1}
        float* wc = wbuf + k % (kPend + 1) * Np;
        float* pb = pbuf + (k & 1) * Np;
        const float tau = R.tau;
        // (B) rows i > k of this CTA: the pending updates of the columns k - pend .. k - 1, then p_i = tau W[i, k+1:] . v.
        // A warp takes kRowsPerWarp rows at a time and a lane issues kLoadsPerRow loads of each before using any, so the
        // pass keeps enough L2 reads in flight to run at bandwidth rather than at L2 latency.
        const int pend = k > 0 ? (k - 1) % kPend + 1 : 0;
        int ov[kPend], ow[kPend];
#pragma unroll
        for (int m = 0; m < kPend; ++m) {
            const int c = max(k - pend + m, 0);
            ov[m] = c % (kPend + 1) * Np;
            ow[m] = (kPend + 1 + c % (kPend + 1)) * Np;
        }
        const int oc = k % (kPend + 1) * Np;
        // row k + 1 as it was last written: nobody writes it in this step, so its loads pass while the rows are at work
        const float* rown = Wb + static_cast<int64_t>(k + 1) * N;
        const int j0 = k + 1 + threadIdx.x;
        float x[kOwnCols];
#pragma unroll
        for (int u = 0; u < kOwnCols; ++u) x[u] = j0 + kSytrdThreads * u < N ? __ldcg(rown + j0 + kSytrdThreads * u) : 0.0f;
        const int i0 = first + wid * C;
        if (pend == 0) update_all<0>(Wb, N, k, i0, nw * C, oc, ov, ow, tau, C, pb);
        else if (pend == kPend) update_all<kPend>(Wb, N, k, i0, nw * C, oc, ov, ow, tau, C, pb);
        else update_all<1>(Wb, N, k, i0, nw * C, oc, ov, ow, tau, C, pb);
        if (first == k + 1) first += C;
        static_assert(kPend == 2, "the cases above");
        cluster_barrier();  // every CTA's p and updated rows are visible
        // (C) w = p - (tau / 2) (p^T v) v over the whole trailing range, and row k + 1 with what is pending and column k's
        // update: the next reflector.  Thread t has the columns k + 1 + t + 512 u of both.
        // Every CTA adds up p^T v from its copy of p in one order whatever the cluster size: `parts` interleaved row sets,
        // each in 16 chains of four rows at a time.
        if (threadIdx.x < 16 * kMaxParts) {
            const int q = threadIdx.x >> 4, chain = threadIdx.x & 15;
            float dot = 0.0f;
            if (q < parts) {
                // set q: rows f, f + parts, ... with f % parts == q
                const int f = k + 1 + (q >= first_dot ? q - first_dot : q - first_dot + parts);
                for (int i = f + chain * kDotRows * parts; i < N; i += 16 * kDotRows * parts) {
                    float pv[kDotRows], vv[kDotRows];
#pragma unroll
                    for (int e = 0; e < kDotRows; ++e) {
                        const int ie = i + e * parts < N ? i + e * parts : i;
                        pv[e] = pb[ie];
                        vv[e] = vc[ie];
                    }
#pragma unroll
                    for (int e = 0; e < kDotRows; ++e)
                        if (i + e * parts < N) dot = fmaf(pv[e], vv[e], dot);
                }
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            if (chain == 0) part[q] = dot;
        }
        if (++first_dot == parts) first_dot = 0;
        __syncthreads();
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < kMaxParts; ++q) {
            const float v = part[q];
            if (q < parts) s += v;
        }
        const float c = -0.5f * tau * s;
        const float vk1 = vc[k + 1], wk1 = fmaf(c, vk1, pb[k + 1]);
        float vp[kPend], wp[kPend];
#pragma unroll
        for (int m = 0; m < kPend; ++m) {
            vp[m] = sm[ov[m] + k + 1];
            wp[m] = sm[ow[m] + k + 1];
        }
        float ss = 0.0f;
#pragma unroll
        for (int u = 0; u < kOwnCols; ++u) {
            const int j = j0 + kSytrdThreads * u;
            if (j >= N) break;
            const float v = vc[j], w = fmaf(c, v, pb[j]);
            wc[j] = w;
#pragma unroll
            for (int m = 0; m < kPend; ++m)
                if (m < pend) x[u] -= __fmul_rn(vp[m], sm[ow[m] + j]) + __fmul_rn(wp[m], sm[ov[m] + j]);
            x[u] -= __fmul_rn(vk1, w) + __fmul_rn(wk1, v);
            if (j == k + 1) scal2[0] = x[u];
            else if (j == k + 2) scal2[1] = x[u];
            else ss = fmaf(x[u], x[u], ss);
        }
        if (r == 0) {  // row k is read by nobody any more: it keeps the reflector
            float* rowv = Wb + static_cast<int64_t>(k) * N;
            for (int j = j0; j < N; j += kSytrdThreads) rowv[j] = vc[j];
            if (threadIdx.x == 0) {
                db[k] = R.d;
                eb[k] = R.beta;
                tb[k] = tau;
            }
        }
        // sum of squares in every thread: the warps' sums, then theirs, as block_sum adds them
        ss = warp_sum(ss);
        float* red_k = red + (k & 1) * 32;
        if (lane == 0) red_k[wid] = ss;
        __syncthreads();
        const float sig = warp_sum(lane < nw ? red_k[lane] : 0.0f);
        if (k + 3 < N) {
            const float alpha = scal2[1];
            Reflector Rn{scal2[0], alpha, 0.0f};
            float scl = 1.0f;
            if (sig > 0.0f) {
                Rn.beta = -copysignf(sqrtf(fmaf(alpha, alpha, sig)), alpha);
                Rn.tau = (Rn.beta - alpha) / Rn.beta;
                scl = 1.0f / (alpha - Rn.beta);
            } else {
                scl = 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kOwnCols; ++u) {
                const int j = j0 + kSytrdThreads * u;
                if (j < N && j > k + 2) vn[j] = x[u] * scl;
            }
            if (threadIdx.x == 0) vn[k + 2] = 1.0f;
            __syncthreads();
            R = Rn;
        } else if (r == 0 && threadIdx.x == 0) {  // k = N - 3: rows N - 2 and N - 1 get column k's update: T's trailing 2 x 2
            auto update = [&](float y, int i, int j, int pending) {
#pragma unroll
                for (int m = 0; m < kPend; ++m)
                    if (m < pending) y -= __fmul_rn(sm[ov[m] + i], sm[ow[m] + j]) + __fmul_rn(sm[ow[m] + i], sm[ov[m] + j]);
                return y - (__fmul_rn(vc[i], wc[j]) + __fmul_rn(wc[i], vc[j]));
            };
            db[N - 2] = update(__ldcg(rown + N - 2), N - 2, N - 2, pend);
            eb[N - 2] = update(__ldcg(rown + N - 1), N - 2, N - 1, pend);
            db[N - 1] = update(__ldcg(Wb + static_cast<int64_t>(N - 1) * N + N - 1), N - 1, N - 1, pend == kPend ? 0 : pend);
        }
    }
    if (r == 0 && threadIdx.x == 0) {
        if (N == 2) {
            db[0] = Wb[0];
            eb[0] = Wb[1];
            db[1] = Wb[N + 1];
        } else if (N == 1) {
            db[0] = Wb[0];
        }
        eb[N - 1] = 0.0f;
        tb[N - 1] = 0.0f;
        if (N >= 2) tb[N - 2] = 0.0f;
    }
    cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

// ---- eigenvalues of T: multisection on Sturm counts ------------------------------------------------------------

// 1 / x by the hardware reciprocal (within 1 ulp; |x| >= pivmin >= 1e-30 is normal here)
__device__ __forceinline__ float rcp_hw(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Numbers of eigenvalues of T below each of K points (FP32, pivots floored at pivmin in magnitude).  The quotient
// e^2 / q takes the hardware reciprocal: the division's full-precision sequence made the search bound by its
// instruction count, and a count from quotients within 1 ulp is the exact count of a T whose e^2 differ by that
// much.  The K recurrences are independent, so their latencies overlap.
template <int K>
__device__ __forceinline__ void sturm_counts(const float* d, const float* e2, int N, const float (&x)[K], float pivmin,
                                             int (&cnt)[K]) {
    float q[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        q[k] = d[0] - x[k];
        if (fabsf(q[k]) < pivmin) q[k] = -pivmin;
        cnt[k] = q[k] < 0.0f;
    }
    for (int i = 1; i < N; ++i) {
        const float di = d[i], ei = e2[i - 1];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            q[k] = (di - x[k]) - ei * rcp_hw(q[k]);
            if (fabsf(q[k]) < pivmin) q[k] = -pivmin;
            cnt[k] += q[k] < 0.0f;
        }
    }
}

// grid (ceil(N / kBisectThreads), batch): eigenvalue j of matrix b into evals[b][j], ascending.  Each step splits
// the bracket at kSectPts equispaced points (multisection: kBisectSteps steps narrow it by 2^-48, as 48 halvings
// would); a thread's recurrences run interleaved, and the small blocks spread the eigenvalues over every SM.
__global__ void __launch_bounds__(kBisectThreads)
k_tridiag_bisect(const float* __restrict__ d_all, const float* __restrict__ e_all, int N, float* __restrict__ evals,
                 float* __restrict__ tnorm_out) {
    extern __shared__ float sm[];
    float* d = sm;
    float* e2 = sm + N;
    __shared__ float red[34];
    const int b = blockIdx.y;
    const float* db = d_all + static_cast<int64_t>(b) * N;
    const float* eb = e_all + static_cast<int64_t>(b) * N;
    float lo = INFINITY, hi = -INFINITY;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const float di = db[i];
        const float el = i > 0 ? fabsf(eb[i - 1]) : 0.0f;
        const float er = i + 1 < N ? fabsf(eb[i]) : 0.0f;
        d[i] = di;
        if (i + 1 < N) e2[i] = eb[i] * eb[i];
        lo = fminf(lo, di - el - er);
        hi = fmaxf(hi, di + el + er);
    }
    // block min / max through warp shuffles
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = lo;
        red[16 + (threadIdx.x >> 5)] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float l = red[0], h = red[16];
        for (int w = 1; w < (blockDim.x >> 5); ++w) {
            l = fminf(l, red[w]);
            h = fmaxf(h, red[16 + w]);
        }
        red[32] = l;
        red[33] = h;
    }
    __syncthreads();
    const float gl = red[32], gu = red[33];
    const float tnorm = fmaxf(fabsf(gl), fabsf(gu));
    if (blockIdx.x == 0 && threadIdx.x == 0) tnorm_out[b] = tnorm;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    const float pivmin = fmaxf(1e-30f, 1.2e-7f * 1e-6f * tnorm);
    float a = gl - 1e-6f * tnorm - 1e-30f, z = gu + 1e-6f * tnorm + 1e-30f;
    // the interval [a, z) holds the (j+1)-th smallest eigenvalue: count(a) <= j < count(z)
    for (int it = 0; it < kBisectSteps; ++it) {
        const float w = z - a;
        float m[kSectPts];
        bool inside = false;
#pragma unroll
        for (int k = 0; k < kSectPts; ++k) {
            m[k] = a + w * (static_cast<float>(k + 1) / static_cast<float>(kSectPts + 1));
            inside |= m[k] > a && m[k] < z;
        }
        if (!inside) break;  // the bracket is down to adjacent floats
        int cnt[kSectPts];
        sturm_counts<kSectPts>(d, e2, N, m, pivmin, cnt);
        // the points rise with k (a + w t is monotone in t), and so do their counts: the lowest point above index j
        // closes the bracket, the highest one at or below it opens it
        float na = a, nz = z;
#pragma unroll
        for (int k = kSectPts - 1; k >= 0; --k)
            if (cnt[k] > j) nz = m[k];
#pragma unroll
        for (int k = 0; k < kSectPts; ++k)
            if (cnt[k] <= j) na = m[k];
        a = na;
        z = nz;
    }
    evals[static_cast<int64_t>(b) * N + j] = 0.5f * (a + z);
}

// ---- eigenvectors of T: inverse iteration in FP64 -------------------------------------------------------------

__device__ __forceinline__ double start_value(int i, int j) {
    uint32_t h = static_cast<uint32_t>(i) * 0x9E3779B1u ^ (static_cast<uint32_t>(j) + 0x7F4A7C15u) * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return 0.5 + static_cast<double>(h & 0xFFFFFF) * (1.0 / 16777216.0);  // in [0.5, 1.5)
}

// grid (ceil(N / 128), batch), one thread per eigenvalue index j.  Scratch S (batch, 3, N, N) FP64: S[0] the
// reciprocal LDL^T pivots 1 / D, S[1] the multipliers L, S[2] the iterate x, element i of thread j at [i * N + j]
// (coalesced over a warp's consecutive j).  Z (batch, N, N) FP32: eigenvector j of T in column j.
//
// Each pass over a vector is a recurrence (one FP64 FMA per element on the previous element's result), so the loads
// it needs are issued kInvitBlock elements ahead into registers: the recurrence then waits only on FMA latency, not
// on a memory round trip per element.  The iterate is normalised lazily: the next solve scales it on the fly.
// Members of a cluster of close eigenvalues get slightly separated shifts (their cluster is orthonormalised after).
__global__ void __launch_bounds__(128)
k_tridiag_invit(const float* __restrict__ d_all, const float* __restrict__ e_all, const float* __restrict__ evals,
                const float* __restrict__ tnorm_all, int N, double* __restrict__ S, float* __restrict__ Z) {
    const int b = blockIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    const float* db = d_all + static_cast<int64_t>(b) * N;
    const float* eb = e_all + static_cast<int64_t>(b) * N;
    const float* lam = evals + static_cast<int64_t>(b) * N;
    const double tnorm = static_cast<double>(tnorm_all[b]);
    const double tol = kClusterTol * tnorm;
    int j0 = j;  // first index of j's cluster
    while (j0 > 0 && static_cast<double>(lam[j0]) - static_cast<double>(lam[j0 - 1]) < tol) --j0;
    const double lm = static_cast<double>(lam[j]) + (j - j0) * 1e-3 * tol;
    const int64_t NN = static_cast<int64_t>(N) * N;
    double* __restrict__ D = S + (static_cast<int64_t>(b) * 3 + 0) * NN + j;
    double* __restrict__ L = S + (static_cast<int64_t>(b) * 3 + 1) * NN + j;
    double* __restrict__ X = S + (static_cast<int64_t>(b) * 3 + 2) * NN + j;
    float* Zb = Z + static_cast<int64_t>(b) * NN;
    const double pivmin = 1e-14 * tnorm + 1e-300;
    constexpr int B = kInvitBlock;
    // LDL^T of T - lm I as the multipliers L and the reciprocal pivots 1 / D, with the first solve's forward pass
    // z_i = x_i - L_{i-1} z_{i-1} on the pseudo-random start x
    double dcur = static_cast<double>(db[0]) - lm;
    if (fabs(dcur) < pivmin) dcur = -pivmin;
    double inv = 1.0 / dcur;
    double z = start_value(0, j);
    D[0] = inv;
    X[0] = z;
    for (int i = 1; i < N; ++i) {
        const double ei = static_cast<double>(eb[i - 1]);
        const double l = ei * inv;
        dcur = (static_cast<double>(db[i]) - lm) - l * ei;
        if (fabs(dcur) < pivmin) dcur = -pivmin;
        inv = 1.0 / dcur;
        z = fma(-l, z, start_value(i, j));
        L[static_cast<int64_t>(i - 1) * N] = l;
        D[static_cast<int64_t>(i) * N] = inv;
        X[static_cast<int64_t>(i) * N] = z;
    }
    double sc = 1.0;  // pending scale of X
    for (int it = 0; it < kInvitSolves; ++it) {
        if (it > 0) {  // forward: z_i = sc x_i - L_{i-1} z_{i-1}
            z = sc * X[0];
            X[0] = z;
            for (int i0 = 1; i0 < N; i0 += B) {
                double xb[B], lb[B];
#pragma unroll
                for (int u = 0; u < B; ++u) {
                    const int i = i0 + u;
                    xb[u] = i < N ? X[static_cast<int64_t>(i) * N] : 0.0;
                    lb[u] = i < N ? L[static_cast<int64_t>(i - 1) * N] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < B; ++u) {
                    const int i = i0 + u;
                    if (i < N) {
                        z = fma(-lb[u], z, sc * xb[u]);
                        X[static_cast<int64_t>(i) * N] = z;
                    }
                }
            }
        }
        // backward: y_i = z_i / D_i - L_i y_{i+1}
        double y = X[static_cast<int64_t>(N - 1) * N] * D[static_cast<int64_t>(N - 1) * N];
        X[static_cast<int64_t>(N - 1) * N] = y;
        double nrm = y * y;
        for (int i0 = N - 2; i0 >= 0; i0 -= B) {
            double xb[B], db2[B], lb[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int i = i0 - u;
                xb[u] = i >= 0 ? X[static_cast<int64_t>(i) * N] : 0.0;
                db2[u] = i >= 0 ? D[static_cast<int64_t>(i) * N] : 0.0;
                lb[u] = i >= 0 ? L[static_cast<int64_t>(i) * N] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int i = i0 - u;
                if (i >= 0) {
                    y = fma(xb[u], db2[u], -lb[u] * y);
                    X[static_cast<int64_t>(i) * N] = y;
                    nrm = fma(y, y, nrm);
                }
            }
        }
        sc = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    }
    for (int i = 0; i < N; ++i) Zb[static_cast<int64_t>(i) * N + j] = static_cast<float>(sc * X[static_cast<int64_t>(i) * N]);
}

// grid (ceil(N / kOrthCols), batch): a block orthonormalises the clusters whose first eigenvalue is among its kOrthCols
// (modified Gram-Schmidt on the columns of Z, lanes over the rows, FP64 sums).  Once column q is final it is taken out of
// every later column of the cluster, a warp per column: each column sees the same subtractions in the same order as it
// would one column after another.  (One warp did all pairs of a cluster in turn: 35 of the 43 ms of a batch of marker
// Grams whose padding repeats one eigenvalue ~100 times.)
constexpr int kOrthThreads = 512, kOrthCols = 16;

__device__ void orth_cluster(float* __restrict__ Zb, int N, int j, int jend, float* pivot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = j; q < jend; ++q) {
        if (warp == 0) {
            double nrm = 0.0;
            for (int i = lane; i < N; i += 32) {
                const double v = static_cast<double>(Zb[static_cast<int64_t>(i) * N + q]);
                nrm = fma(v, v, nrm);
            }
            nrm = warp_sum(nrm);
            const double sc = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
            for (int i = lane; i < N; i += 32) {
                float* zq = Zb + static_cast<int64_t>(i) * N + q;
                const float v = static_cast<float>(sc * static_cast<double>(*zq));
                *zq = v;
                pivot[i] = v;
            }
        }
        __syncthreads();
        for (int m = q + 1 + warp; m < jend; m += kOrthThreads / 32) {
            double pr = 0.0;
#pragma unroll 4
            for (int i = lane; i < N; i += 32)
                pr = fma(static_cast<double>(pivot[i]), static_cast<double>(Zb[static_cast<int64_t>(i) * N + m]), pr);
            pr = warp_sum(pr);
#pragma unroll 4
            for (int i = lane; i < N; i += 32) {
                float* zm = Zb + static_cast<int64_t>(i) * N + m;
                *zm = static_cast<float>(static_cast<double>(*zm) - pr * static_cast<double>(pivot[i]));
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kOrthThreads)
k_cluster_orth(const float* __restrict__ evals, const float* __restrict__ tnorm_all, int N, float* __restrict__ Z) {
    extern __shared__ float pivot[];  // one column
    __shared__ int end_s[kOrthCols];  // end of the cluster that starts at each of the block's columns, 0 if none does
    const int b = blockIdx.y, j0 = blockIdx.x * kOrthCols;
    if (threadIdx.x < kOrthCols) {
        const int j = j0 + threadIdx.x;
        const float* lam = evals + static_cast<int64_t>(b) * N;
        const double tol = kClusterTol * static_cast<double>(tnorm_all[b]);
        auto close = [&](int i) { return static_cast<double>(lam[i]) - static_cast<double>(lam[i - 1]) < tol; };
        int e = 0;
        if (j < N && !(j > 0 && close(j))) {
            e = j + 1;
            while (e < N && close(e)) ++e;
            if (e - j < 2) e = 0;
        }
        end_s[threadIdx.x] = e;
    }
    __syncthreads();
    for (int c = 0; c < kOrthCols; ++c)
        if (end_s[c]) orth_cluster(Z + static_cast<int64_t>(b) * N * N, N, j0 + c, end_s[c], pivot);
}

// ---- back-transformation: U = Q Z with Q = H_0 ... H_{N-3} in WY blocks ---------------------------------------

// grid (nblocks, batch), kWy * kWy threads: T_q of block q (upper triangular, I - V T V^T = H_{k0} ... H_{k0+15}),
// from G = V^T V and tau (LAPACK larft, forward / columnwise)
__global__ void __launch_bounds__(kWy * kWy)
k_wy_factors(const float* __restrict__ W, const float* __restrict__ tau_all, int N, int n_refl,
             float* __restrict__ Tq) {
    __shared__ float G[kWy][kWy + 1];
    __shared__ float T[kWy][kWy + 1];
    const int b = blockIdx.y, q = blockIdx.x;
    const int k0 = q * kWy;
    const int a = threadIdx.x / kWy, c = threadIdx.x % kWy;
    const float* Wb = W + static_cast<int64_t>(b) * N * N;
    const float* tau = tau_all + static_cast<int64_t>(b) * N;
    const int ka = k0 + a, kc = k0 + c;
    float g = 0.0f;
    if (a < c && kc < n_refl) {  // v_a . v_c over rows > kc (v_c is zero above row kc + 1, where it is 1)
        const float* va = Wb + static_cast<int64_t>(ka) * N;
        const float* vc = Wb + static_cast<int64_t>(kc) * N;
        g = va[kc + 1];
        for (int i = kc + 2; i < N; ++i) g = fmaf(va[i], vc[i], g);
    }
    G[a][c] = g;
    T[a][c] = 0.0f;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kWy; ++i) {
            const float ti = (k0 + i < n_refl) ? tau[k0 + i] : 0.0f;
            // T[0:i, i] = -ti * T[0:i, 0:i] G[0:i, i]
            for (int rr = 0; rr < i; ++rr) {
                float s = 0.0f;
                for (int m = rr; m < i; ++m) s = fmaf(T[rr][m], G[m][i], s);
                T[rr][i] = -ti * s;
            }
            T[i][i] = ti;
        }
    }
    __syncthreads();
    Tq[((static_cast<int64_t>(b) * gridDim.x + q) * kWy + a) * kWy + c] = T[a][c];
}

// grid (ceil(N / kTile), batch): columns c0 .. c0 + kTile - 1 of Z (eigenvectors of T) to eigenvector rows of A in U.
//
// Every entry of S = V^T Z is one chain of multiply-adds down the rows, every entry of Z -= V S' one over the block's
// reflectors.  Round q goes down the rows once: Z -= V_q S'_q a chunk ahead of S_{q-1} = V_{q-1}^T Z, the one by four
// warps with the 16 x 4 entries of S' of a thread's columns in registers, the other by two with 2 x 2 chains a thread;
// both blocks' rows come through a ring of kRing chunks.  Shared-memory reads and a barrier a chunk bound it.  One phase after
// the other, an operand read per multiply-add and a chunk's loads waited for: 20 x 1,000 x 1,000 4.20 -> 2.61 ms, 8 x 1,600 x
// 1,600 7.98 -> 4.61.
template <int kTile>
struct Bt {
    static constexpr int kDot = 4 * kTile;             // threads of V^T Z
    static constexpr int kUpd = 8 * kTile;             // and of Z -= V S'
    static constexpr int kThreads = kDot + kUpd;
    static constexpr int kMaxN = kTile == 16 ? kSytrdThreads * kOwnCols : 1900;
    static constexpr size_t smem(int N) {
        return sizeof(float) * (static_cast<size_t>(N + kChunk) * kTile + kRing * 2 * kWy * kChunk);
    }
};
static_assert(Bt<16>::smem(Bt<16>::kMaxN) <= 222 * 1024 && Bt<24>::smem(Bt<24>::kMaxN) <= 222 * 1024, "shared memory budget");

template <int kTile>
__global__ void __launch_bounds__(Bt<kTile>::kThreads, kTile == 16 ? 2 : 1)
k_backtransform(const float* __restrict__ W, const float* __restrict__ Tq_all, const float* __restrict__ Z, int N,
                int n_refl, int nblocks, float* __restrict__ U) {
    constexpr int kBtThreads = Bt<kTile>::kThreads, kBtDot = Bt<kTile>::kDot, kUpd = Bt<kTile>::kUpd;
    extern __shared__ float4 sm4[];
    float* Zt = reinterpret_cast<float*>(sm4);  // N x kTile, kChunk rows of zeros
    float* ring = Zt + (N + kChunk) * kTile;    // kRing x [V_q, V_{q-1}] x kWy x kChunk
    __shared__ float Sm[kWy][kTile + 1];
    __shared__ __align__(16) float Sp[kWy][kTile];  // -S'
    __shared__ float Tm[kWy][kWy + 1];
    const int b = blockIdx.y;
    const int c0 = blockIdx.x * kTile;
    const int64_t NN = static_cast<int64_t>(N) * N;
    const float* Wb = W + b * NN;
    const float* Zb = Z + b * NN;
    const float* Tb = Tq_all + static_cast<int64_t>(b) * nblocks * kWy * kWy;
    const int ncols = min(kTile, N - c0);
    const int tid = threadIdx.x;
    // rows base(q) + kChunk j .. of blocks q and q - 1, by the threads of the second phase: into registers, and an iteration
    // later to ring slot j (rows of a block from its first one on)
    constexpr int kEntries = 2 * kWy * kChunk, kPre = (kEntries + kUpd - 1) / kUpd;
    float pre[kPre];
    auto base = [&](int q) { return max(q - 1, 0) * kWy + 1; };
    constexpr int kStep = kUpd / kChunk;  // reflectors la, la + kStep, ..., of both blocks one after the other, row li
    static_assert(kUpd % kChunk == 0, "a thread's entries of a chunk are of one row");
    const int la = (tid - kBtDot) / kChunk, li = (tid - kBtDot) % kChunk;
    auto load = [&](int q, int j) {
        const int i0 = base(q) + j * kChunk, i = i0 + li;
        if (j > 0 && q > 0 && (q + 1) * kWy <= n_refl && i0 + kChunk <= N) {  // nothing to leave out
#pragma unroll
            for (int u = 0; u < kPre; ++u) {
                const int a = min(la + u * kStep, 2 * kWy - 1);
                pre[u] = Wb[(q * kWy + a - (a < kWy ? 0 : 2 * kWy)) * N + i];
            }
            return;
        }
#pragma unroll
        for (int u = 0; u < kPre; ++u) {
            const int a = la + u * kStep, k = q * kWy + a - (a < kWy ? 0 : 2 * kWy);
            pre[u] = (a < 2 * kWy && i < N && k >= 0 && k < n_refl && i > k) ? Wb[k * N + i] : 0.0f;
        }
    };
    auto store = [&](int j) {
        float* slot = ring + (j % kRing) * kEntries;
#pragma unroll
        for (int u = 0; u < kPre; ++u) {
            const int t = tid - kBtDot + u * kUpd;
            if (kEntries % kUpd == 0 || t < kEntries) slot[t] = pre[u];
        }
    };
    if (tid >= kBtDot) {
        load(nblocks, 0);
        store(0);
        load(nblocks, 1);
    }
    for (int t = tid; t < (N + kChunk) * kTile; t += kBtThreads) {
        const int i = t / kTile, c = t % kTile;
        Zt[t] = c < ncols && i < N ? Zb[static_cast<int64_t>(i) * N + c0 + c] : 0.0f;
    }
    // S: reflectors sa, sa + 1 and columns sc, sc + 1 of a thread of the first phase
    const int sa = tid / (kTile / 2) * 2, sc = tid % (kTile / 2) * 2;
    // Z -= V S': columns zc .. zc + 3 of a chunk's rows zr and zr + 32 of a thread of the other warps
    constexpr int kQuads = kTile / 4;
    static_assert(kUpd / kQuads == kChunk / 2, "two rows of four columns a thread");
    const int zc = (tid - kBtDot) % kQuads * 4, zr = (tid - kBtDot) / kQuads;
    for (int q = nblocks; q >= 0; --q) {
        const int i0 = base(q), first = q * kWy + 1;  // first row that V_q touches
        const int chunks = (N - i0 + kChunk - 1) / kChunk;
        float s[2][2] = {};
        float4 ns[kWy] = {};
        if (tid >= kBtDot && q < nblocks) {
#pragma unroll
            for (int m = 0; m < kWy; ++m) ns[m] = *reinterpret_cast<const float4*>(&Sp[m][zc]);
        }
        if (q > 0)
            for (int t = tid; t < kWy * kWy; t += kBtThreads)
                Tm[t / kWy][t % kWy] = Tb[static_cast<int64_t>(q - 1) * kWy * kWy + t];
        for (int j = 0; j <= chunks; ++j) {
            __syncthreads();  // chunk j is staged, and rows of chunk j - 1 are up to date
            if (tid >= kBtDot) {
                if (j + 1 < chunks) store(j + 1);
                if (j + 2 < chunks) load(q, j + 2);
                else if (j + 2 == max(chunks, 2) && q > 0) load(q - 1, 0);
                if (j == chunks || q == nblocks) continue;
                const float* V = ring + (j % kRing) * 2 * kWy * kChunk;
                const int r = i0 + j * kChunk, end = min(kChunk, N - r);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ii = zr + h * (kChunk / 2);
                    if (ii >= end || r + ii < first) continue;
                    float4* zp = reinterpret_cast<float4*>(Zt + (r + ii) * kTile + zc);
                    float4 z = *zp;
#pragma unroll
                    for (int m = 0; m < kWy; ++m) {
                        const float v = V[m * kChunk + ii];
                        z.x = fmaf(v, ns[m].x, z.x);
                        z.y = fmaf(v, ns[m].y, z.y);
                        z.z = fmaf(v, ns[m].z, z.z);
                        z.w = fmaf(v, ns[m].w, z.w);
                    }
                    *zp = z;
                }
            } else if (j > 0 && q > 0) {
                // eight rows at a time, the next eight on their way (rows past N are zeros in both operands)
                const float* v = ring + ((j - 1) % kRing) * 2 * kWy * kChunk + (kWy + sa) * kChunk;
                const float* z = Zt + (i0 + (j - 1) * kChunk) * kTile + sc;
                float4 vv[2][2][2];  // [buffer][reflector][rows / 4]
                float2 zz[2][8];
                auto fetch = [&](int u, int ii) {
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int h = 0; h < 2; ++h) vv[u][a][h] = *reinterpret_cast<const float4*>(v + a * kChunk + ii + 4 * h);
#pragma unroll
                    for (int e = 0; e < 8; ++e) zz[u][e] = *reinterpret_cast<const float2*>(z + (ii + e) * kTile);
                };
                fetch(0, 0);
#pragma unroll
                for (int g = 0; g < kChunk / 8; ++g) {
                    if (g + 1 < kChunk / 8) fetch((g + 1) & 1, 8 * (g + 1));
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float2 x = zz[g & 1][e];
#pragma unroll
                        for (int a = 0; a < 2; ++a) {
                            const float4 f = vv[g & 1][a][e / 4];
                            const float y = e % 4 == 0 ? f.x : e % 4 == 1 ? f.y : e % 4 == 2 ? f.z : f.w;
                            s[a][0] = fmaf(y, x.x, s[a][0]);
                            s[a][1] = fmaf(y, x.y, s[a][1]);
                        }
                    }
                }
            }
        }
        if (q == 0) break;
        if (tid < kBtDot) {
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                Sm[sa + a][sc] = s[a][0];
                Sm[sa + a][sc + 1] = s[a][1];
            }
        }
        __syncthreads();
        if (tid >= kBtDot) {
            store(0);
            load(q - 1, 1);
        }
        // S' = T S
        for (int t = tid; t < kWy * kTile; t += kBtThreads) {
            const int a = t / kTile, cc = t % kTile;
            float sp = 0.0f;
#pragma unroll
            for (int m = 0; m < kWy; ++m) sp = m >= a ? fmaf(Tm[a][m], Sm[m][cc], sp) : sp;
            Sp[a][cc] = -sp;
        }
        __syncthreads();
    }
    __syncthreads();
    // eigenvector c0 + c is column c of the tile: one row of U each
    for (int c = 0; c < ncols; ++c)
        for (int i = tid; i < N; i += kBtThreads) U[b * NN + static_cast<int64_t>(c0 + c) * N + i] = Zt[i * kTile + c];
}

template <int kTile>
int launch_backtransform(const float* W, const float* Tq, const float* Z, int N, int n_refl, int nblocks, int batch, float* U,
                         cudaStream_t st) {
    const size_t smem = Bt<kTile>::smem(N);
    // (per device, so set on every call, to one bound whatever N, so that another host thread's call never lowers it under
    // this launch; the call is cheap)
    FLMM_CUDA(cudaFuncSetAttribute(k_backtransform<kTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(Bt<kTile>::smem(Bt<kTile>::kMaxN))));
    k_backtransform<kTile><<<dim3(ceil_div(N, kTile), batch), Bt<kTile>::kThreads, smem, st>>>(W, Tq, Z, N, n_refl, nblocks, U);
    return check_launch("k_backtransform");
}

struct OwnLayout {
    size_t W, Z, S, d, e, tau, ev, tn, T, total;
    int nblocks;
};

// Clusters of each size that fit on the device at once (one CTA per SM; a cluster lies within one GPC, so 7 CTAs fit 15
// times on 152 SMs where 6 fit 23 times), and the size with the least time for a batch: waves of clusters times the
// column's row pass, shared by the cluster, plus what does not shrink (barrier, reductions, the next reflector).
int cluster_ctas(int dev, int N, int batch, int* out) {
    static std::mutex mu;
    static int active[64][kMaxClusterCtas + 1];
    static bool known[64];
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64) return fail(FLMM_ERR_ARG, "eigh: device %d", dev);
    // (per device context, so set on every call; the calls are cheap)
    FLMM_CUDA(cudaFuncSetAttribute(k_sytrd_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    FLMM_CUDA(cudaFuncSetAttribute(k_sytrd_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (!known[dev]) {
        for (int c = 2; c <= kMaxClusterCtas; ++c) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = static_cast<unsigned>(c);
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(static_cast<unsigned>(c * 64));
            cfg.blockDim = dim3(kSytrdThreads);
            cfg.dynamicSmemBytes = 96 * 1024;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k_sytrd_cluster, &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            }
            active[dev][c] = n;
        }
        known[dev] = true;
    }
    const double rows = kRowPassCycles * (N / 1000.0) * (N / 1000.0);
    double best = 0.0;
    *out = 0;
    for (int c = 2; c <= kMaxClusterCtas; ++c) {
        if (active[dev][c] < 1) continue;
        const double waves = (batch + active[dev][c] - 1) / active[dev][c];
        const double cost = waves * (rows / c + kColumnCycles + kCtaCycles * c);
        if (*out == 0 || cost < best) {
            best = cost;
            *out = c;
        }
    }
    return *out ? FLMM_OK : fail(FLMM_ERR_CUDA, "eigh: no cluster of the tridiagonalisation fits on the device");
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

OwnLayout own_layout(int N, int batch) {
    OwnLayout L;
    const size_t NN = static_cast<size_t>(N) * N * batch;
    const int n_refl = N > 2 ? N - 2 : 0;
    L.nblocks = n_refl > 0 ? (n_refl + kWy - 1) / kWy : 0;
    size_t o = 0;
    L.W = o; o += up256(4 * NN);
    L.Z = o; o += up256(4 * NN);
    L.S = o; o += up256(8 * 3 * NN);
    L.d = o; o += up256(4 * static_cast<size_t>(N) * batch);
    L.e = o; o += up256(4 * static_cast<size_t>(N) * batch);
    L.tau = o; o += up256(4 * static_cast<size_t>(N) * batch);
    L.ev = o; o += up256(4 * static_cast<size_t>(N) * batch);
    L.tn = o; o += up256(4 * static_cast<size_t>(batch));
    L.T = o; o += up256(4 * static_cast<size_t>(L.nblocks > 0 ? L.nblocks : 1) * kWy * kWy * batch);
    L.total = o;
    return L;
}

}  // namespace

namespace flmm {

size_t eigh_own_workspace_bytes(int N, int batch) { return own_layout(N, batch).total; }

// A (batch, N, N) FP32 symmetric in, eigenvector rows out (ascending eigenvalues into evals (batch, N) FP32)
int eigh_own_f32(float* A, int N, int batch, float* evals, void* work, cudaStream_t st) {
    const OwnLayout L = own_layout(N, batch);
    char* base = static_cast<char*>(work);
    float* W = reinterpret_cast<float*>(base + L.W);
    float* Z = reinterpret_cast<float*>(base + L.Z);
    double* S = reinterpret_cast<double*>(base + L.S);
    float* d = reinterpret_cast<float*>(base + L.d);
    float* e = reinterpret_cast<float*>(base + L.e);
    float* tau = reinterpret_cast<float*>(base + L.tau);
    float* tn = reinterpret_cast<float*>(base + L.tn);
    float* Tq = reinterpret_cast<float*>(base + L.T);
    const size_t NN = static_cast<size_t>(N) * N;
    FLMM_CUDA(cudaMemcpyAsync(W, A, 4 * NN * batch, cudaMemcpyDeviceToDevice, st));
    // 1. tridiagonalisation, one cluster per matrix
    const int Np = (N + 3) & ~3;
    const size_t smem1 = sizeof(float) * ((2 * kPend + 4) * static_cast<size_t>(Np) + 64 + kMaxParts + 2);
    int dev = 0, sms = 0;
    FLMM_CUDA(cudaGetDevice(&dev));
    FLMM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // the row sets that p^T v is added up in: part of the result, so they follow the batch and not the cluster
    const int parts = std::max(2, std::min(kMaxParts, sms / std::max(batch, 1)));
    int C = 0;
    int rc = cluster_ctas(dev, N, batch, &C);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(C);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(C * batch), 1, 1);
    cfg.blockDim = dim3(kSytrdThreads, 1, 1);
    cfg.dynamicSmemBytes = smem1;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FLMM_CUDA(cudaLaunchKernelEx(&cfg, k_sytrd_cluster, W, N, parts, d, e, tau));
    if ((rc = check_launch("k_sytrd_cluster"))) return rc;
    // 2. eigenvalues
    k_tridiag_bisect<<<dim3(ceil_div(N, kBisectThreads), batch), kBisectThreads,
                       sizeof(float) * 2 * static_cast<size_t>(N), st>>>(
        d, e, N, evals, tn);
    if ((rc = check_launch("k_tridiag_bisect"))) return rc;
    // 3. eigenvectors of T
    k_tridiag_invit<<<dim3(ceil_div(N, kInvitThreads), batch), kInvitThreads, 0, st>>>(d, e, evals, tn, N, S, Z);
    if ((rc = check_launch("k_tridiag_invit"))) return rc;
    k_cluster_orth<<<dim3(ceil_div(N, kOrthCols), batch), kOrthThreads, sizeof(float) * N, st>>>(evals, tn, N, Z);
    if ((rc = check_launch("k_cluster_orth"))) return rc;
    // 4. back-transformation into A
    const int n_refl = N > 2 ? N - 2 : 0;
    if (L.nblocks > 0) {
        k_wy_factors<<<dim3(L.nblocks, batch), kWy * kWy, 0, st>>>(W, tau, N, n_refl, Tq);
        if ((rc = check_launch("k_wy_factors"))) return rc;
    }
    // Two CTAs of 16 columns an SM as long as they fit; then one of 24, as long as that fits (8 x 1,600 x 1,600: 4.61 ms, one
    // of 16 5.61); then one of 16.
    if (N <= 1310) return launch_backtransform<16>(W, Tq, Z, N, n_refl, L.nblocks, batch, A, st);
    if (N <= Bt<24>::kMaxN) return launch_backtransform<24>(W, Tq, Z, N, n_refl, L.nblocks, batch, A, st);
    return launch_backtransform<16>(W, Tq, Z, N, n_refl, L.nblocks, batch, A, st);
}

}  // namespace flmm
