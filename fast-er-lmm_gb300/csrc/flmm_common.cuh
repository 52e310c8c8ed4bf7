// Shared helpers of the fasterlmm_gb300 CUDA library: status handling, argument checks, warp reductions and the
// FP64 atomic max used by the per-column genome max.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fasterlmm_gb300.h"

namespace flmm {

// Records a printf-style message as this thread's last error (read back by flmm_last_error) and returns `status`.
int fail(int status, const char* fmt, ...);

// Counts one kernel launch of this library and converts the pending CUDA error (if any) into FLMM_ERR_CUDA with
// the kernel's name.  Call once right after each <<<...>>> launch.
int check_launch(const char* what);

// Same error conversion without counting a launch (after library calls such as cuSOLVER).
int check_cuda(const char* what);

// Device int raised by kernels without a context (e.g. the refinement's tensor-core product) when a bounded wait
// gives up; one per device, allocated on first use, reported and cleared by flmm_context_check.  nullptr if the
// allocation failed.
int* device_err_flag(int device);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// tcgen05 kernel form: CTA pairs unless FLMM_TC_PAIR=0 asks for the single-CTA kernels (kept for cross-checks).
bool use_pair_kernels();

// The library's own batched FP32 eigensolver (csrc/flmm_eigh_own.cu): A (batch, N, N) symmetric in, one eigenvector
// per row out, evals (batch, N) ascending; work of eigh_own_workspace_bytes(N, batch) bytes.
size_t eigh_own_workspace_bytes(int N, int batch);
int eigh_own_f32(float* A, int N, int batch, float* evals, void* work, cudaStream_t st);

// The refinement's FP64-accurate product on the tensor cores (csrc/flmm_ozaki.cu): W (batch, N, N) = U~ A^T, U~ the
// digit-plane rounding of U (written to Ut); work of refine_product_tc_bytes(N, batch) bytes.
size_t refine_product_tc_bytes(int N, int batch);
int refine_product_tc(const float* U, const double* A, int N, int batch, float* Ut, double* W, void* work,
                      cudaStream_t st);
// The step's corrections on the same workspace, after refine_product_tc: M = U~ R^T, then U_out = U~ + T U~ with T
// (batch, N, N) FP32 stored at the start of the workspace and scratch an (batch, N, N) FP32 buffer.
int refine_m_tc(const float* R, int N, int batch, float* M, void* work, cudaStream_t st);
int refine_update_tc(const float* T, const float* Ut, float* scratch, int N, int batch, float* U_out, void* work,
                     cudaStream_t st);

// flmm_project_kinship of n_units stacked kinships in place (csrc/flmm_prep.cu).
size_t project_kinships_bytes(int N, int D, int n_units);
int project_kinships(double* K, const double* Qx, int N, int D, int n_units, void* work, cudaStream_t st);

// flmm_mean_f32 and flmm_wald_interp_nodes of n_units stacked spectra: shat (n_units), W (n_units, R, Neff)
// (csrc/flmm_fast.cu).
int interp_units(const double* s, int Neff, int n_units, float* shat, double x0, double h, int R, double* W,
                 cudaStream_t st);

// One unit of a grouped split product: tiles of A rows [a_row0, a_row0 + a_rows) against B rows [b_row0, b_row0 + b_rows),
// numbered from tile0 on (256 A rows x 128 B rows, csrc/flmm_fast.cu).
struct UnitTiles {
    int tile0, a_row0, a_rows, b_row0, b_rows;
};
constexpr int kUnitTileA = 256, kUnitTileB = 128;

// Grouped launches over the units of a scan (csrc/flmm_fast.cu).  units: device array of n_units; total: all tiles.
// units_pair_ok: whether grouped launches may run (the pair kernels are available and no other form is forced).
bool units_pair_ok();
// C[a row][b row - b_row0] = A B^T for every unit's rows, over K.
int gemm_units(flmm_context* ctx, const void* Ah, const void* Al, const float* sa, int64_t lda, int a_total, const void* Bh,
               const void* Bl, const float* sb, int64_t ldb, int b_total, int K, float* C, int64_t ldc,
               const UnitTiles* units, int n_units, int total, cudaStream_t st);
// The fused Wald of flmm_wald_split_f16 with the columns of unit u in rows u P .. of the column operands and variants in
// rows of their own; listed tests hold the variant's row.  largest: the unit whose shape the tile order is tuned on.
struct WaldUnits {
    const void *A1h, *A1l;
    int64_t lda;
    const float* sa1;
    const void *Lh, *Ll;
    int64_t ldl;
    const float *sl, *rWr, *rWr0;
    int P, n_real, n_units;
    const void *B1h, *B1l;
    int64_t ldb;
    const float* sb1;
    const void *Fh, *Fl;
    int64_t ldf;
    const float* sf;
    int M, Neff, R;
    const int64_t* rows;
    double *f, *beta, *se, *sfve;
    int64_t ldo;
    double* max_F;
    float f_refine;
    int32_t *flag_count, *flags;
    int flag_cap;
};
int wald_units(flmm_context* ctx, const WaldUnits& w, const UnitTiles* units, int total, const UnitTiles& largest,
               cudaStream_t st);
// flmm_split_rows_f16 of n_units stacked FP32 matrices: rows of X from x_stride entries apart into rows dst_rows apart.
int split_units(const float* X, int64_t ldx, int64_t x_stride, int rows, int K, int n_units, void* hi, void* lo, int64_t ldo,
                int dst_rows, float* scale, cudaStream_t st);
// flmm_wald_split_prep_columns of every unit: s32 (n_units, Neff), UY uy_stride entries apart, log delta (n_units, P),
// outputs with unit u's columns from row u P on.
int prep_columns_units(const float* s32, int Neff, const float* UYt, int64_t ldu, int64_t uy_stride, const double* log_delta,
                       int P, int n_units, const float* shat, double x0, double h, int R, void* A1h, void* A1l, int64_t lda,
                       void* Lh, void* Ll, int64_t ldl, float* sa1, float* sl, float* rWr, float* rWr0, cudaStream_t st);
// flmm_fit_delta_fast of every unit (csrc/flmm_delta_fast.cu): s (n_units, Neff), log_delta and idx (n_units, P).
size_t fit_units_bytes(int Neff, int n_grid, int n_units);
int fit_delta_units(const double* s, int Neff, const float* UYt, int64_t ldu, int64_t uy_stride, int P, int n_units,
                    int n_grid, double lo, double hi, int refine, double* log_delta, int32_t* idx, void* work,
                    cudaStream_t st);
// flmm_wald_refine_f32 of every unit (csrc/flmm_wald_refine.cu): variant rows over all units, unit u's from start[u] on
// (device, n_units + 1 entries).
int wald_refine_units(flmm_context* ctx, const int32_t* flags, const int32_t* flag_count, int flag_cap, float f_refine,
                      const float* US, int64_t ldus, const float* UYt, int64_t ldu, int64_t uy_stride, const float* s32,
                      const double* log_delta, int P, int Neff, int M, int n_real, const int* start, int n_units,
                      const int64_t* rows, double* f, double* beta, double* se, double* sfve, int64_t ldo, double* max_F,
                      cudaStream_t st);
// flmm_fill_nullh2 of every unit (csrc/flmm_prep.cu).
int fill_nullh2_units(const double* log_delta, int P, int n_real, const int64_t* rows, const int* start, int n_units,
                      int most, double* out, int64_t ldo, cudaStream_t st);

// SMs of the current device
inline int sm_count(int* out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(out, cudaDevAttrMultiProcessorCount, dev);
    return e == cudaSuccess ? FLMM_OK : fail(FLMM_ERR_CUDA, "sm_count: %s", cudaGetErrorString(e));
}

inline unsigned ceil_div(int64_t a, int64_t b) { return static_cast<unsigned>((a + b - 1) / b); }

#define FLMM_REQUIRE(cond, ...)                                                       \
    do {                                                                              \
        if (!(cond)) return ::flmm::fail(FLMM_ERR_ARG, __VA_ARGS__);                  \
    } while (0)

#define FLMM_CUDA(call)                                                               \
    do {                                                                              \
        cudaError_t e_ = (call);                                                      \
        if (e_ != cudaSuccess)                                                        \
            return ::flmm::fail(FLMM_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The golden-section bracket of the reference (fasterlmm/core.py:545-558), in its operations; [grid[i-1], grid[i+1]] first.
struct Bracket {
    double a, b, inv_phi, inv_phi2;

    __device__ Bracket(const double* grid, int G, int i)
        : a(grid[max(i - 1, 0)]), b(grid[min(i + 1, G - 1)]), inv_phi(2.0 / (1.0 + sqrt(5.0))) {
        inv_phi2 = __dmul_rn(inv_phi, inv_phi);
    }
    __device__ double c() const { return __dadd_rn(a, __dmul_rn(inv_phi2, __dadd_rn(b, -a))); }
    __device__ double d() const { return __dadd_rn(a, __dmul_rn(inv_phi, __dadd_rn(b, -a))); }
    __device__ void narrow(bool left) {
        const double nc = c(), nd = d();
        b = left ? nd : b;
        a = left ? a : nc;
    }
    // The step after losses (c, d).  Of the next two points one is an old one but for its rounding: whether point e is the
    // old one to the bit, and its loss.
    __device__ bool narrow_kept(const double* loss, int e, double* kept) {
        const double oc = c(), od = d(), lc = loss[0], ld = loss[1];
        const bool left = lc < ld;
        narrow(left);
        *kept = left ? lc : ld;
        return left ? e == 1 && d() == oc : e == 0 && c() == od;
    }
};

// Neumaier-compensated running sum: comp collects the rounding error of every addition, so sum + comp is the sum of
// the added terms without the accumulated FP32 rounding
__device__ __forceinline__ void neumaier(float& sum, float& comp, float x) {
    const float t = sum + x;
    comp += (fabsf(sum) >= fabsf(x)) ? ((sum - t) + x) : ((x - t) + sum);
    sum = t;
}

// exact sum and error of a + b (Knuth's TwoSum)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// warp-wide sum of a compensated pair (hi + lo), TwoSum at every level of the butterfly
__device__ __forceinline__ float warp_sum_pair(float hi, float lo) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, hi, o);
        const float ol = __shfl_xor_sync(0xffffffffu, lo, o);
        float sum, err;
        two_sum(hi, oh, sum, err);
        hi = sum;
        lo = lo + ol + err;
    }
    return hi + lo;
}

__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// max over non-negative (or NaN) doubles stored as their bit patterns: for x >= 0 the IEEE bit pattern read as a
// signed 64-bit integer is monotone in x, -inf (the initial value) reads negative, and NaN reads above +inf, so
// a NaN column statistic propagates as torch.maximum would.
__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
    atomicMax(reinterpret_cast<long long*>(addr), __double_as_longlong(v));
}

__device__ __forceinline__ void atomic_max_nonneg(float* addr, float v) {
    atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));
}

// FP64 helpers that are never contracted into an FMA, so an expression evaluates with the same roundings as the
// reference's separate tensor operations.
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// Positive clamp floor of the FP64 path (fasterlmm/core.py:80-86).
constexpr double kPosFloor = 1e-300;

}  // namespace flmm
