// FP64 SIMT GEMM of the plain (FP64-faithful) form: the per-chromosome Gram that builds every LOCO kinship
// (fasterlmm/io.py:257-265) and the eigenbasis rotations (fasterlmm/core.py:518, :629).  GB300's FP64 pipe (two
// multiply-adds per cycle and SM) is the bound, far below shared memory's rate even at one output per thread, so the
// tile is chosen for an even load of the SMs alone: tiles of (16 R) x (16 R) outputs, R = 4, 2 or 1, next stage's
// elements in registers while a stage is used.  Every output is one chain of multiply-adds over k whatever the tile, so
// the tile does not change a bit.  A Gram A A^T forms its lower tiles and mirrors them (a product of two numbers does not
// depend on their order).  Against 64 x 64 tiles throughout: a 1,000-marker Gram over 20,000 samples 40 -> 20 ms, the
// products of a low-rank scan of 2,000 samples 45 -> 18 ms.
#include "flmm_common.cuh"
#include "flmm_oz64.cuh"

using namespace flmm;

namespace {

constexpr int BK = 16, NT = 256;

// C (Mr, Nr) = alpha * sum_k A(i, k) B(j, k) + beta * C.  A(i, k) is A[i * lda + k] when AK (k contiguous), else
// A[k * lda + i]; likewise B.  Thread (tx, ty) of the 16 x 16 block owns rows i0 + ty + 16 r and columns
// j0 + tx + 16 c, so stores of consecutive tx hit consecutive columns.  SYM: blocks are the tiles on and below the
// diagonal of A A^T, numbered row by row.
template <bool AK, bool BK_CONTIG, int R, bool SYM>
__global__ void __launch_bounds__(NT)
k_gemm_f64(const double* __restrict__ A, int64_t lda, const double* __restrict__ B, int64_t ldb, double* __restrict__ C,
           int64_t ldc, int Mr, int Nr, int K, double alpha, double beta) {
    constexpr int T = 16 * R;
    __shared__ double As[BK][T + 1];
    __shared__ double Bs[BK][T + 1];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    int bi = blockIdx.y, bj = blockIdx.x;
    if (SYM) {
        const int t = blockIdx.x;
        bi = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
        while (bi * (bi + 1) / 2 > t) --bi;
        while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
        bj = t - bi * (bi + 1) / 2;
    }
    const int i0 = bi * T, j0 = bj * T;
    double va[R], vb[R];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int l = 0; l < R; ++l) {
            const int t = tid + l * NT;
            const int ia = AK ? t / BK : t % T, ka = AK ? t % BK : t / T;
            const int ib = BK_CONTIG ? t / BK : t % T, kb = BK_CONTIG ? t % BK : t / T;
            const int gi = i0 + ia, gj = j0 + ib;
            va[l] = (gi < Mr && k0 + ka < K)
                        ? (AK ? A[static_cast<int64_t>(gi) * lda + k0 + ka] : A[static_cast<int64_t>(k0 + ka) * lda + gi])
                        : 0.0;
            vb[l] = (gj < Nr && k0 + kb < K) ? (BK_CONTIG ? B[static_cast<int64_t>(gj) * ldb + k0 + kb]
                                                          : B[static_cast<int64_t>(k0 + kb) * ldb + gj])
                                             : 0.0;
        }
    };
    double acc[R][R] = {};
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int l = 0; l < R; ++l) {
            const int t = tid + l * NT;
            As[AK ? t % BK : t / T][AK ? t / BK : t % T] = va[l];
            Bs[BK_CONTIG ? t % BK : t / T][BK_CONTIG ? t / BK : t % T] = vb[l];
        }
        __syncthreads();
        if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            double a[R], b[R];
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = As[k][ty + 16 * r];
#pragma unroll
            for (int c = 0; c < R; ++c) b[c] = Bs[k][tx + 16 * c];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < R; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
        }
        __syncthreads();
    }
    auto store = [&](int gi, int gj, double x) {
        double* dst = C + static_cast<int64_t>(gi) * ldc + gj;
        const double v = alpha * x;
        *dst = (beta == 0.0) ? v : v + beta * (*dst);
    };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int gi = i0 + ty + 16 * r;
        if (gi >= Mr) continue;
#pragma unroll
        for (int c = 0; c < R; ++c) {
            const int gj = j0 + tx + 16 * c;
            if (gj >= Nr || (SYM && gj > gi)) continue;
            store(gi, gj, acc[r][c]);
            if (SYM && gj != gi) store(gj, gi, acc[r][c]);
        }
    }
}

// The tile whose fullest SM has the least to do; each halving of the tile costs a few percent in loads.
template <bool AK, bool BKC, bool SYM>
int launch_gemm(const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc, int Mr, int Nr, int K,
                double alpha, double beta, cudaStream_t st, const char* what) {
    int sm = 0;
    const int rc = sm_count(&sm);
    if (rc) return rc;
    auto tiles = [&](int r) {
        const int64_t ti = ceil_div(Mr, 16 * r), tj = ceil_div(Nr, 16 * r);
        return SYM ? ti * (ti + 1) / 2 : ti * tj;
    };
    int best = 4;
    double cost = 0.0;
    for (int r = 4; r >= 1; r /= 2) {
        if (!SYM && ceil_div(Mr, 16 * r) > 65535u) break;  // grid limit
        const double c = static_cast<double>((tiles(r) + sm - 1) / sm) * r * r * (r == 4 ? 1.0 : r == 2 ? 1.03 : 1.12);
        if (r == 4 || c < cost) {
            cost = c;
            best = r;
        }
    }
    const dim3 grid = SYM ? dim3(static_cast<unsigned>(tiles(best))) : dim3(ceil_div(Nr, 16 * best), ceil_div(Mr, 16 * best));
    auto go = [&](auto kernel) { kernel<<<grid, NT, 0, st>>>(A, lda, B, ldb, C, ldc, Mr, Nr, K, alpha, beta); };
    if (best == 4) go(k_gemm_f64<AK, BKC, 4, SYM>);
    else if (best == 2) go(k_gemm_f64<AK, BKC, 2, SYM>);
    else go(k_gemm_f64<AK, BKC, 1, SYM>);
    return check_launch(what);
}

}  // namespace

extern "C" int flmm_gemm_nt_f64(const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
                                int Mr, int Nr, int K, double alpha, void* stream) {
    FLMM_REQUIRE(A && B && C && Mr >= 0 && Nr >= 0 && K >= 0 && lda >= K && ldb >= K && ldc >= Nr,
                 "flmm_gemm_nt_f64: bad arguments");
    if (Mr == 0 || Nr == 0) return FLMM_OK;
    if (A == B && lda == ldb && Mr == Nr)
        return launch_gemm<true, true, true>(A, lda, B, ldb, C, ldc, Mr, Nr, K, alpha, 0.0, as_stream(stream),
                                             "k_gemm_f64<nt, symmetric>");
    return launch_gemm<true, true, false>(A, lda, B, ldb, C, ldc, Mr, Nr, K, alpha, 0.0, as_stream(stream),
                                          "k_gemm_f64<nt>");
}

namespace {

// Rows of one operand digitised at a time: digit planes of at most 256 MB (16 bytes per element).
int oz_block(int rows, int unit, int K) {
    const size_t fit = (size_t(256) << 20) / (16 * static_cast<size_t>(K)) / unit * unit;
    if (fit < static_cast<size_t>(unit)) return unit;
    return fit < static_cast<size_t>(rows) ? static_cast<int>(fit) : rows;
}

}  // namespace

extern "C" int flmm_gemm_nt_f64_tc_workspace_bytes(int Mr, int Nr, int K, size_t* bytes) {
    FLMM_REQUIRE(bytes && Mr >= 0 && Nr >= 0 && K > 0, "flmm_gemm_nt_f64_tc_workspace_bytes: bad arguments");
    *bytes = oz_operand_bytes(oz_block(Mr, kOzRowsA, K), K, 1, kOzRowsA) +
             oz_operand_bytes(oz_block(Nr, kOzRowsB, K), K, 1, kOzRowsB) + 1024;
    return FLMM_OK;
}

extern "C" int flmm_gemm_nt_f64_tc(const double* A, int64_t lda, const double* B, int64_t ldb, const double* D,
                                   int64_t ldd, double* C, int64_t ldc, int Mr, int Nr, int K, void* work,
                                   size_t work_bytes, void* stream) {
    FLMM_REQUIRE(A && B && C && work && Mr >= 0 && Nr >= 0 && K > 0 && lda >= K && ldb >= K && ldc >= Nr &&
                     (!D || ldd >= Nr),
                 "flmm_gemm_nt_f64_tc: bad arguments");
    size_t need = 0;
    flmm_gemm_nt_f64_tc_workspace_bytes(Mr, Nr, K, &need);
    if (work_bytes < need)
        return fail(FLMM_ERR_WORKSPACE, "flmm_gemm_nt_f64_tc: need %zu bytes, got %zu", need, work_bytes);
    if (Mr == 0 || Nr == 0) return FLMM_OK;
    cudaStream_t st = as_stream(stream);
    const int ra = oz_block(Mr, kOzRowsA, K), rb = oz_block(Nr, kOzRowsB, K);
    char* wa = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(work) + 1023) / 1024 * 1024);
    char* wb = wa + oz_operand_bytes(ra, K, 1, kOzRowsA);
    for (int j0 = 0; j0 < Nr; j0 += rb) {
        const OzOperand b = oz_carve(wb, Nr - j0 < rb ? Nr - j0 : rb, K, 1, kOzRowsB);
        int rc = oz_digits(b, 0, B + j0 * ldb, ldb, false, nullptr, 0, st);
        if (rc) return rc;
        for (int i0 = 0; i0 < Mr; i0 += ra) {
            const OzOperand a = oz_carve(wa, Mr - i0 < ra ? Mr - i0 : ra, K, 1, kOzRowsA);
            if ((rc = oz_digits(a, 0, A + i0 * lda, lda, false, nullptr, 0, st))) return rc;
            const OzProduct p{A + i0 * lda, lda, 0, B + j0 * ldb, ldb, {false, false}, OzGate::kPlain, C + i0 * ldc + j0, ldc, 0,
                              D ? D + i0 * ldd + j0 : nullptr, ldd};
            if ((rc = oz_gemm(a, b, p, st))) return rc;
        }
    }
    return FLMM_OK;
}

extern "C" int flmm_gram_f64(const double* Zt, int64_t ldzt, int M, int N, double beta, double* Gc, int64_t ldg,
                             void* stream) {
    FLMM_REQUIRE(Zt && Gc && M >= 0 && N > 0 && ldzt >= N && ldg >= N, "flmm_gram_f64: bad arguments");
    if (M == 0 && beta != 0.0) return FLMM_OK;
    return launch_gemm<false, false, true>(Zt, ldzt, Zt, ldzt, Gc, ldg, N, N, M, 1.0, beta, as_stream(stream),
                                           "k_gemm_f64<gram>");
}
