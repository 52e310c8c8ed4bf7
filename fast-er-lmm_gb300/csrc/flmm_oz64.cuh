// FP64 products C = A B^T on the FP16 tensor cores from exact digit planes (csrc/flmm_oz64.cu): the interface used by
// the FP64 Wald scans and the rotations of tested variants.
#pragma once

#include <cuda_fp16.h>

#include "flmm_common.cuh"

namespace flmm {

constexpr int kOzPlanes = 8;      // 7-bit digit planes per operand (55 bits below the row's leading bit)
constexpr int kOzRowsA = 128;     // A rows per tile
constexpr int kOzRowsB = 64;      // B rows per tile

// One operand: `batches` stacked matrices of (rows, K) as digit planes, row exponents and tile qualities.  A row keeps
// the eight digits of every 16 elements together, [k / 16][plane][k % 16], so that a stage of the product reads 256
// contiguous bytes of it (zeros from K to the next multiple of 16).
struct OzOperand {
    __half* planes;   // [batch][row][ldp]
    int* expo;        // [batch][row]
    float* mean;      // [batch][row]: mean |x| over 2^expo
    float* qual;      // [batch][tile]: largest quality of a tile's rows (oz_digits), infinity where digits cannot hold a row
    int* err;         // of an operand A: [0] set once a product with it gave up a wait, [1] once one had tiles that digits
                      // do not hold; zeroed with its batch 0's digits
    int64_t ldp;
    int rows, K, batches, tile_rows;
    int tiles() const { return (rows + tile_rows - 1) / tile_rows; }
};

size_t oz_operand_bytes(int rows, int K, int batches, int tile_rows);
OzOperand oz_carve(void* base, int rows, int K, int batches, int tile_rows);

// Balancing exponents of a product's reduction: e_k of the size that |X[., k]| usually reaches over the rows of X (pitch
// ldx); bal holds oz_balance_ints(K) ints, e_k in the first K.  A product's operands may be digitised as A 2^e_k and
// B 2^-e_k (both squared where B is): the digits then resolve each term against the largest term that the variants leave
// possible at k, not against an entry of A that meets zeros.  e_k is the median of the largest finite entries of
// kOzBalanceGroups groups of rows: the largest over all rows would let one variant's outlier set the resolution of every
// column for all the others, and the median entry follows the sample too loosely (rows then spread half as far again).
constexpr int kOzBalanceGroups = 15;
inline size_t oz_balance_ints(int K) { return (1 + kOzBalanceGroups) * static_cast<size_t>(K); }
int oz_balance(const double* X, int64_t ldx, int rows, int K, int* bal, cudaStream_t st);

// Digits of batch `b` of `op` from the rows of X (pitch ldx), or of their squares, times 2^(times bal_k).  A row's quality
// is its largest |x| over the root of its mean square, over its mean |x| where it is balanced, or with `weights` over the
// root of the mean of row r / per of the weights' batch 1 (balanced by twice `times`).
struct OzWeights {
    const OzOperand* op;
    int per;
};
int oz_digits(const OzOperand& op, int b, const double* X, int64_t ldx, bool square, const int* bal, int times,
              cudaStream_t st, OzWeights weights = {nullptr, 0});

// What a product's tiles must fulfil for their digits to be used (see quality_limit).
enum class OzGate {
    kPlain,     // unbalanced operands
    kBalanced,  // balanced operands; batches of squares are sums of non-negative terms
    kTerms      // terms whose squares are taken from the weighted sums: A's digits with weights, B's balanced
};

// C[b] (rows of A, rows of B; pitch ldc, batch stride c_stride) = A[b] B[b]^T, or D - A B^T where D is given (pitch
// ldd).  Xa, Xb: the FP64 matrices the digits were taken from (Xa with a batch stride; Xb shared by the batches, its
// elements squared in batch b where square[b] is set), read where a tile's digits are not good enough, and for all tiles
// where the kernel gave up one of its bounded waits or CTA pairs are not to be had (FLMM_TC_PAIR=0, or none fits).
// Operands may hold more batches than the product takes; it takes the smaller count, from batch 0.
struct OzProduct {
    const double* Xa;
    int64_t lda, xa_stride;
    const double* Xb;
    int64_t ldb;
    bool square[2];
    OzGate gate;
    double* C;
    int64_t ldc, c_stride;
    const double* D;
    int64_t ldd;
};
int oz_gemm(const OzOperand& A, const OzOperand& B, const OzProduct& p, cudaStream_t st);

// The Wald epilogue over the sums of P columns x Mc variants (flmm_wald_f64.cu), pitch ldg: a column's sWy in its row of
// Gy, sWs in its row of Gs, and in the GLS form the nq terms whose squares add to B^T A^-1 B in nq rows of Gq (nq = 0 in
// the compat form).  F, beta, SE, SFVE of the first n_real columns into rows `rows` of the outputs, column maxima into
// max_F.
int wald_finish(const double* Gy, const double* Gs, const double* Gq, int nq, int64_t ldg, const double* rWr,
                double var_df, int P, int n_real, int Mc, const int64_t* rows, double* f, double* beta, double* se,
                double* sfve, int64_t ldo, double* max_F, cudaStream_t st);

// Products below this many multiply-adds stay on the FP64 pipe.
bool oz_worth(int64_t Mr, int64_t Nr, int64_t K);

}  // namespace flmm
