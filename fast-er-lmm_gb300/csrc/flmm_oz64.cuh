// FP64 products C = A B^T on the FP16 tensor cores from exact digit planes (csrc/flmm_oz64.cu): the interface used by
// the FP64 Wald scans and the rotations of tested variants.
#pragma once

#include <cuda_fp16.h>

#include "flmm_common.cuh"

namespace flmm {

constexpr int kOzPlanes = 8;      // 7-bit digit planes per operand (55 bits below the row's leading bit)
constexpr int kOzRowsA = 128;     // A rows per tile
constexpr int kOzRowsB = 64;      // B rows per tile

// One operand: `batches` stacked matrices of (rows, K) as digit planes, row exponents and tile qualities.
struct OzOperand {
    __half* planes;   // [plane][batch][row][ldp]
    int* expo;        // [batch][row]
    float* qual;      // [batch][tile]: largest max|x| / rms(x) of a tile's rows, infinity where digits cannot hold a row
    int64_t ldp;
    int rows, K, batches, tile_rows;
    int tiles() const { return (rows + tile_rows - 1) / tile_rows; }
};

size_t oz_operand_bytes(int rows, int K, int batches, int tile_rows);
OzOperand oz_carve(void* base, int rows, int K, int batches, int tile_rows);

// Digits of batch `b` of `op` from the rows of X (pitch ldx), or of their squares.
int oz_digits(const OzOperand& op, int b, const double* X, int64_t ldx, bool square, cudaStream_t st);

// C[b] (rows of A, rows of B; pitch ldc, batch stride c_stride) = A[b] B[b]^T, or D - A B^T where D is given (pitch
// ldd).  Xa, Xb: the FP64 matrices the digits were taken from (batch strides xa_stride, xb_stride; batch 1 of Xb is
// the squares of Xb itself where square_b1 is set), read where a tile's digits are not good enough.
struct OzProduct {
    const double* Xa;
    int64_t lda, xa_stride;
    const double* Xb;
    int64_t ldb, xb_stride;
    bool square_b1;
    double* C;
    int64_t ldc, c_stride;
    const double* D;
    int64_t ldd;
};
int oz_gemm(const OzOperand& A, const OzOperand& B, const OzProduct& p, cudaStream_t st);

// Products below this many multiply-adds stay on the FP64 pipe.
bool oz_worth(int64_t Mr, int64_t Nr, int64_t K);

}  // namespace flmm
