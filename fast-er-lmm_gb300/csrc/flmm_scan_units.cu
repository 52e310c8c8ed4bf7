// The fast form's chromosome work issued from native code on caller-owned buffers: what fasterlmm_gb300.fast.scan_t runs.
//
//   flmm_loco_kinships_f32   per-chromosome Grams of a kinship panel (split-FP16 tensor-core products), the LOCO kinships
//                            of every unit and their projection off the covariates
//   flmm_scan_units          every unit's column side (eigenvector split, UY rotation, delta fit) and variant side (US
//                            rotation, Wald operands, fused Wald, strong-test re-evaluation, nullh2), the column side of
//                            unit u + 1 on a second stream beside the variant side of unit u
//
// Each unit is ~20 launches of a few microseconds for ordinary studies, and issuing them from Python cost 10-20 us each:
// 150 samples x 1,500 variants on 16 chromosomes took 10.2 ms in 505 launches, 4.35 unit by unit and 3.00 grouped.  What
// depends on the spectra alone (mean, FP32 copies, sWs node weights and their split) and the projections run for all units
// in one launch each.  Where every unit's operands fit kGroupBytes together, so does the rest (run_grouped): the launches
// then take all units' rows, the split products with the units' tiles one after another.  The arithmetic is in every form
// that of the C entry points called one by one.
#include <cuda_fp16.h>
#include <limits.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <vector>

#include "flmm_common.cuh"

using namespace flmm;

namespace {

constexpr double kInterpH = 0.25;  // sWs interpolation nodes in log delta (see flmm_wald_split_prep_columns)
constexpr int kInterpQ = 10;

inline int64_t pad8(int64_t k) { return (k + 7) / 8 * 8; }

// Carves a workspace; with a null base it only adds up sizes.
struct Arena {
    char* base;
    size_t off = 0;
    explicit Arena(void* p) : base(reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 1023) / 1024 * 1024)) {}
    void* take(size_t bytes) {
        void* p = base + off;
        off += (bytes + 1023) / 1024 * 1024;
        return p;
    }
    template <typename T>
    T* of(size_t n) { return static_cast<T*>(take(sizeof(T) * (n > 0 ? n : 1))); }
};

struct SplitBuf {
    __half *hi, *lo;
    float* scale;
    int64_t ld;
};

SplitBuf take_split(Arena& a, int64_t rows, int64_t ld) {
    SplitBuf s;
    s.hi = a.of<__half>(static_cast<size_t>(rows) * ld);
    s.lo = a.of<__half>(static_cast<size_t>(rows) * ld);
    s.scale = a.of<float>(rows);
    s.ld = ld;
    return s;
}

int interp_nodes(double lo, double hi, double* x0) {
    *x0 = lo - (kInterpQ / 2) * kInterpH;
    return static_cast<int>(std::ceil((hi - lo) / kInterpH - 1e-9)) + kInterpQ + 1;
}

// ---- LOCO kinships ----------------------------------------------------------------------------------------------

// y[t] = x_0[t] + x_1[t] + ... in FP64, the n FP32 arrays one after another
__global__ void k_sum_grams(const float* __restrict__ x, int64_t len, int n, double* __restrict__ y) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (t >= len) return;
    double s = 0.0;
    for (int i = 0; i < n; ++i) s += static_cast<double>(x[i * len + t]);
    y[t] = s;
}

constexpr int kPut = 256;
template <typename T>
struct Put {
    T x[kPut];
};
template <typename T>
__global__ void k_put(Put<T> p, int n, T* __restrict__ to) {
    if (static_cast<int>(threadIdx.x) < n) to[threadIdx.x] = p.x[threadIdx.x];
}

// A host table into device memory, as launch parameters: it needs no buffer that outlives the call, also under capture.
template <typename T>
int put(const T* from, int n, T* to, cudaStream_t st) {
    static_assert(sizeof(Put<T>) <= 24000, "launch parameters");
    for (int i = 0; i < n; i += kPut) {
        Put<T> p = {};
        const int k = std::min(kPut, n - i);
        std::copy(from + i, from + i + k, p.x);
        k_put<T><<<1, kPut, 0, st>>>(p, k, to + i);
        int rc = check_launch("k_put");
        if (rc) return rc;
    }
    return FLMM_OK;
}

struct UnitGram {
    int block;      // the unit's own chromosome among the panel's, or -1
    double m_loco;  // variants in its kinship
};

__global__ void k_unit_kinships(const double* __restrict__ Gtot, const float* __restrict__ grams, int64_t nn,
                                const UnitGram* __restrict__ units, double* __restrict__ K) {
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (t >= nn) return;
    const UnitGram u = units[blockIdx.y];
    const double own = u.block >= 0 ? static_cast<double>(grams[u.block * nn + t]) : 0.0;
    K[blockIdx.y * nn + t] = (Gtot[t] - own) / u.m_loco;
}

}  // namespace

extern "C" int flmm_loco_kinships_f32_workspace_bytes(int N, int D, int n_blocks, const int* counts, int n_units,
                                                      size_t* bytes) {
    FLMM_REQUIRE(bytes && N > 0 && D > 0 && n_blocks >= 0 && (counts || n_blocks == 0) && n_units > 0,
                 "flmm_loco_kinships_f32_workspace_bytes: bad arguments");
    int64_t mpad = 0;
    for (int c = 0; c < n_blocks; ++c) mpad += (counts[c] + 63) / 64 * 64;
    mpad = std::max<int64_t>(mpad, 64);
    const size_t proj = project_kinships_bytes(N, D, n_units);
    Arena a(nullptr);
    a.of<double>(static_cast<size_t>(N) * mpad);
    take_split(a, N, mpad);
    a.of<float>(static_cast<size_t>(N) * N * n_blocks);
    a.of<double>(static_cast<size_t>(N) * N);
    a.of<UnitGram>(n_units);
    a.take(proj);
    *bytes = a.off + 2048;
    return FLMM_OK;
}

extern "C" int flmm_loco_kinships_f32(flmm_context* ctx, const double* Zt, int N, const int* counts, int n_blocks,
                                      const int* unit_block, int n_units, const double* Qx, int D, double* Kp, void* work,
                                      size_t work_bytes, void* stream) {
    FLMM_REQUIRE(ctx && Zt && counts && unit_block && Qx && Kp && work && N > 0 && D > 0 && n_blocks > 0 && n_units > 0,
                 "flmm_loco_kinships_f32: bad arguments");
    size_t need = 0;
    int rc = flmm_loco_kinships_f32_workspace_bytes(N, D, n_blocks, counts, n_units, &need);
    if (rc) return rc;
    if (work_bytes < need)
        return fail(FLMM_ERR_WORKSPACE, "flmm_loco_kinships_f32: need %zu bytes, got %zu", need, work_bytes);
    int64_t M = 0, mpad = 0;
    for (int c = 0; c < n_blocks; ++c) {
        M += counts[c];
        mpad += (counts[c] + 63) / 64 * 64;
    }
    mpad = std::max<int64_t>(mpad, 64);
    for (int u = 0; u < n_units; ++u) {
        FLMM_REQUIRE(unit_block[u] < n_blocks, "flmm_loco_kinships_f32: bad block");
        FLMM_REQUIRE(M - (unit_block[u] >= 0 ? counts[unit_block[u]] : 0) > 0,
                     "flmm_loco_kinships_f32: unit %d holds every kinship variant", u);
    }
    cudaStream_t st = as_stream(stream);
    const int64_t nn = static_cast<int64_t>(N) * N;
    Arena a(work);
    double* Zg = a.of<double>(static_cast<size_t>(N) * mpad);
    const SplitBuf sp = take_split(a, N, mpad);
    float* grams = a.of<float>(static_cast<size_t>(nn) * n_blocks);
    double* Gtot = a.of<double>(nn);
    UnitGram* units = a.of<UnitGram>(n_units);
    void* proj = a.take(project_kinships_bytes(N, D, n_units));
    // sample-major panel, each chromosome's columns from a multiple of 64 on
    FLMM_CUDA(cudaMemsetAsync(Zg, 0, sizeof(double) * N * mpad, st));
    int64_t row = 0, off = 0;
    for (int c = 0; c < n_blocks; ++c) {
        if (counts[c] && (rc = flmm_transpose_f64(Zt + row * N, N, counts[c], N, Zg + off, mpad, stream))) return rc;
        row += counts[c];
        off += (counts[c] + 63) / 64 * 64;
    }
    if ((rc = flmm_split_rows_f16(Zg, 1, mpad, N, static_cast<int>(mpad), sp.hi, sp.lo, mpad, sp.scale, stream))) return rc;
    off = 0;
    for (int c = 0; c < n_blocks; ++c) {
        if ((rc = flmm_gemm_split_f16(ctx, sp.hi + off, sp.lo + off, sp.scale, mpad, N, sp.hi + off, sp.lo + off, sp.scale,
                                      mpad, N, counts[c], grams + c * nn, N, 0, stream)))
            return rc;
        off += (counts[c] + 63) / 64 * 64;
    }
    k_sum_grams<<<ceil_div(nn, 256), 256, 0, st>>>(grams, nn, n_blocks, Gtot);
    if ((rc = check_launch("k_sum_grams"))) return rc;
    try {
        std::vector<UnitGram> host(n_units);
        for (int u = 0; u < n_units; ++u)
            host[u] = UnitGram{unit_block[u], static_cast<double>(M - (unit_block[u] >= 0 ? counts[unit_block[u]] : 0))};
        if ((rc = put(host.data(), n_units, units, st))) return rc;
    } catch (const std::bad_alloc&) {
        return fail(FLMM_ERR_ARG, "flmm_loco_kinships_f32: out of host memory");
    }
    k_unit_kinships<<<dim3(ceil_div(nn, 256), n_units), 256, 0, st>>>(Gtot, grams, nn, units, Kp);
    if ((rc = check_launch("k_unit_kinships"))) return rc;
    return project_kinships(Kp, Qx, N, D, n_units, proj, st);
}

// ---- units ------------------------------------------------------------------------------------------------------

namespace {

// Grouped launches when every unit's column operands (eigenvectors, rotated phenotypes and their weighted rows) take at
// most this much together, and the variants' (rotations and their halves) too: 150 x 1,500 on 16 chromosomes 4.35 -> 3.00
// ms, 563 x 20,011 on 22 15.1 -> 12.5, 1,600 x 6,000 on 8 169 -> 162.  With more columns a unit's launches fill the device
// for many waves, and the second stream hides the rest.
constexpr size_t kGroupBytes = size_t{1} << 30;

struct UnitBufs {
    bool grouped;
    double* s;       // (units, Neff)
    float *s32, *shat;
    double* W;       // (units, R, Neff) sWs node weights
    SplitBuf Ws;
    struct Slot {
        SplitBuf Us;
        float* UY;
        int32_t* idx;
        void* fit;
    } slot[2];
    size_t fit_bytes;
    // grouped: every unit's tiles of the three products and first variant row; rotated phenotypes are (P, units ldk)
    UnitTiles *tiles_us, *tiles_f, *tiles_w;
    int* start;
    float* US;
    __half *A1h, *A1l, *Lh, *Ll, *B1h, *B1l, *B2h, *B2l;
    float *sa1, *sl, *rWr, *rWr0, *sb1, *sb2, *F;
    SplitBuf Fs;
    int32_t *flags, *flag_count;
    int R, cap;
    int64_t ldk, ldr;
    double x0;
};

int carve_units(Arena& a, const flmm_units* q, bool group, UnitBufs* b) {
    const int Neff = q->N - q->D;
    const size_t P = q->P, U = q->n_units;
    int mc = 0;
    for (int u = 0; u < q->n_units; ++u) mc = std::max(mc, q->unit_count[u]);
    b->ldk = pad8(Neff);
    b->R = interp_nodes(q->opts.log_delta_min, q->opts.log_delta_max, &b->x0);
    b->ldr = pad8(b->R);
    b->s = a.of<double>(U * Neff);
    b->s32 = a.of<float>(U * Neff);
    b->shat = a.of<float>(U);
    b->W = a.of<double>(U * b->R * Neff);
    b->Ws = take_split(a, static_cast<int64_t>(U) * b->R, b->ldk);
    int rc = flmm_fit_delta_fast_workspace_bytes(Neff, q->opts.n_grid, &b->fit_bytes);
    if (rc) return rc;
    // one unit's row after another's, and few enough columns
    int64_t total = 0;
    bool dense = group && U > 1 && U <= 32767;  // (grid.y)
    for (int u = 0; u < q->n_units; ++u) {
        dense = dense && q->unit_start[u] == total;
        total += q->unit_count[u];
    }
    const size_t columns = U * b->ldk * 4 * (pad8(q->N) + 2 * P);
    const size_t variants = static_cast<size_t>(total) * (12 * b->ldk + 4 * (b->ldr + pad8(b->R)));
    b->grouped = dense && total < (int64_t{1} << 30) && U * std::max<size_t>(P, b->ldk) < (size_t{1} << 30) &&
                 columns <= kGroupBytes && variants <= kGroupBytes;
    if (b->grouped) {
        UnitBufs::Slot& s = b->slot[0];
        s.Us = take_split(a, static_cast<int64_t>(U) * b->ldk, pad8(q->N));
        s.UY = a.of<float>(U * P * b->ldk);
        s.idx = a.of<int32_t>(U * P);
        s.fit = a.take(fit_units_bytes(Neff, q->opts.n_grid, q->n_units));
        for (UnitTiles** t : {&b->tiles_us, &b->tiles_f, &b->tiles_w}) *t = a.of<UnitTiles>(U);
        b->start = a.of<int>(U + 1);
    } else {
        for (auto& s : b->slot) {
            s.Us = take_split(a, Neff, pad8(q->N));
            s.UY = a.of<float>(P * b->ldk);
            s.idx = a.of<int32_t>(P);
            s.fit = a.take(b->fit_bytes);
        }
    }
    const size_t M = b->grouped ? total : mc;
    const size_t PA = b->grouped ? U * P : P;
    b->US = a.of<float>(M * b->ldk);
    b->A1h = a.of<__half>(PA * b->ldk);
    b->A1l = a.of<__half>(PA * b->ldk);
    b->Lh = a.of<__half>(PA * b->ldr);
    b->Ll = a.of<__half>(PA * b->ldr);
    for (float** x : {&b->sa1, &b->sl, &b->rWr, &b->rWr0}) *x = a.of<float>(PA);
    for (__half** x : {&b->B1h, &b->B1l, &b->B2h, &b->B2l}) *x = a.of<__half>(M * b->ldk);
    for (float** x : {&b->sb1, &b->sb2}) *x = a.of<float>(M);
    b->F = a.of<float>(M * b->ldr);
    b->Fs = take_split(a, M, pad8(b->R));
    const int64_t tests = static_cast<int64_t>(M) * q->n_real;
    const int64_t most = q->refine_cap * (b->grouped ? std::min<int64_t>(q->n_units, 16) : 1);
    b->cap = q->opts.f_refine > 0.0 ? static_cast<int>(std::min<int64_t>({tests, most, INT_MAX / 2})) : 0;
    b->flags = a.of<int32_t>(2 * static_cast<size_t>(b->cap));
    b->flag_count = a.of<int32_t>(1);
    return FLMM_OK;
}

// s[u] = kept spectrum of unit u (fasterlmm/core.py:512-515), its FP32 copy
__global__ void k_unit_spectra(const double* __restrict__ evals, int N, int D, double* __restrict__ s,
                               float* __restrict__ s32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, u = blockIdx.y, Neff = N - D;
    if (i >= Neff) return;
    const double v = fmax(evals[static_cast<int64_t>(u) * N + D + i] - 1.0, 0.0);
    s[static_cast<int64_t>(u) * Neff + i] = v;
    s32[static_cast<int64_t>(u) * Neff + i] = static_cast<float>(v);
}

struct Events {
    cudaEvent_t e[5] = {};
    int make() {
        for (cudaEvent_t& x : e)
            if (cudaEventCreateWithFlags(&x, cudaEventDisableTiming) != cudaSuccess)
                return fail(FLMM_ERR_CUDA, "flmm_scan_units: cannot create an event");
        return FLMM_OK;
    }
    ~Events() {
        for (cudaEvent_t x : e)
            if (x) cudaEventDestroy(x);
    }
};

int check_units(const flmm_units* q) {
    // (F has N - D - 1 degrees of freedom; a grid of one value, log_delta_min = log_delta_max, fixes delta)
    FLMM_REQUIRE(q && q->N > q->D + 1 && q->D >= 1 && q->P >= 0 && q->n_real >= 0 && q->n_real <= q->P && q->n_units > 0 &&
                     q->unit_start && q->unit_count && q->opts.n_grid >= 1 && std::isfinite(q->opts.log_delta_min) &&
                     std::isfinite(q->opts.log_delta_max) && q->refine_cap >= 0 &&
                     q->opts.log_delta_max - q->opts.log_delta_min < 1e8,
                 "flmm_scan_units: bad arguments");
    double x0 = 0.0;
    FLMM_REQUIRE(interp_nodes(q->opts.log_delta_min, q->opts.log_delta_max, &x0) >= kInterpQ,
                 "flmm_scan_units: log_delta_max below log_delta_min");
    for (int u = 0; u < q->n_units; ++u)
        FLMM_REQUIRE(q->unit_start[u] >= 0 && q->unit_count[u] >= 0, "flmm_scan_units: bad unit %d", u);
    return FLMM_OK;
}

int unit_columns(flmm_context* ctx, const flmm_units* q, const UnitBufs& b, int u, cudaStream_t st) {
    const UnitBufs::Slot& s = b.slot[u & 1];
    const int N = q->N, Neff = N - q->D;
    const float* rows = q->U + static_cast<int64_t>(u) * N * N + static_cast<int64_t>(q->D) * N;
    int rc = flmm_split_rows_f16(rows, 0, N, Neff, N, s.Us.hi, s.Us.lo, s.Us.ld, s.Us.scale, st);
    if (rc || q->P == 0) return rc;
    if ((rc = flmm_gemm_split_f16(ctx, q->Yh, q->Yl, q->Yscale, q->ldY, q->P, s.Us.hi, s.Us.lo, s.Us.scale, s.Us.ld, Neff,
                                  N, s.UY, b.ldk, 0, st)))
        return rc;
    return flmm_fit_delta_fast(b.s + static_cast<int64_t>(u) * Neff, Neff, s.UY, b.ldk, q->P, q->opts.n_grid,
                               q->opts.log_delta_min, q->opts.log_delta_max, q->opts.refine,
                               q->log_delta + static_cast<int64_t>(u) * q->P, s.idx, s.fit, b.fit_bytes, st);
}

int unit_variants(flmm_context* ctx, const flmm_units* q, const UnitBufs& b, int u, cudaStream_t st) {
    const int Mc = q->unit_count[u];
    if (Mc == 0) return FLMM_OK;
    const UnitBufs::Slot& s = b.slot[u & 1];
    const int N = q->N, Neff = N - q->D, P = q->P;
    const int64_t a = q->unit_start[u];
    const uint16_t* zh = static_cast<const uint16_t*>(q->Zh) + a * q->ldZ;
    const uint16_t* zl = static_cast<const uint16_t*>(q->Zl) + a * q->ldZ;
    const double* ld = q->log_delta + static_cast<int64_t>(u) * P;
    const int64_t* rows = q->rows + a;
    const float* s32 = b.s32 + static_cast<int64_t>(u) * Neff;
    int rc;
    if ((rc = flmm_gemm_split_f16(ctx, zh, zl, q->Zscale + a, q->ldZ, Mc, s.Us.hi, s.Us.lo, s.Us.scale, s.Us.ld, Neff, N,
                                  b.US, b.ldk, 0, st)))
        return rc;
    if ((rc = flmm_wald_split_prep_columns(s32, Neff, s.UY, b.ldk, ld, P, b.shat + u, b.x0, kInterpH, b.R, b.A1h, b.A1l,
                                           b.ldk, b.Lh, b.Ll, b.ldr, b.sa1, b.sl, b.rWr, b.rWr0, st)))
        return rc;
    if ((rc = flmm_wald_split_prep_variants(b.US, b.ldk, Mc, Neff, b.B1h, b.B1l, b.B2h, b.B2l, b.ldk, b.sb1, b.sb2, st)))
        return rc;
    // node values of sWs~: F (Mc, R) = (US o US) W~^T
    const int64_t w0 = static_cast<int64_t>(u) * b.R;
    if ((rc = flmm_gemm_split_f16(ctx, b.B2h, b.B2l, b.sb2, b.ldk, Mc, b.Ws.hi + w0 * b.ldk, b.Ws.lo + w0 * b.ldk,
                                  b.Ws.scale + w0, b.ldk, b.R, Neff, b.F, b.ldr, 0, st)))
        return rc;
    if ((rc = flmm_split_rows_f16(b.F, 0, b.ldr, Mc, b.R, b.Fs.hi, b.Fs.lo, b.Fs.ld, b.Fs.scale, st))) return rc;
    const bool refine = q->opts.f_refine > 0.0 && q->n_real > 0;
    const int cap = refine ? static_cast<int>(std::min<int64_t>(static_cast<int64_t>(Mc) * q->n_real, b.cap)) : 0;
    const float cut = refine ? static_cast<float>(q->opts.f_refine) : INFINITY;
    if ((rc = flmm_wald_split_f16(ctx, b.A1h, b.A1l, b.ldk, b.sa1, b.Lh, b.Ll, b.ldr, b.sl, b.rWr, b.rWr0, P, q->n_real,
                                  b.B1h, b.B1l, b.ldk, b.sb1, b.Fs.hi, b.Fs.lo, b.Fs.ld, b.Fs.scale, Mc, Neff, b.R, rows,
                                  q->f, q->beta, q->se, q->sfve, q->ldo, q->max_F, cut, refine ? b.flag_count : nullptr,
                                  refine ? b.flags : nullptr, cap, st)))
        return rc;
    if (refine && (rc = flmm_wald_refine_f32(ctx, b.flags, b.flag_count, cap, cut, b.US, b.ldk, s.UY, b.ldk, s32, ld, Neff, Mc,
                                             q->n_real, rows, q->f, q->beta, q->se, q->sfve, q->ldo, q->max_F, st)))
        return rc;
    return flmm_fill_nullh2(ld, q->n_real, rows, Mc, q->nullh2, q->ldo, st);
}

// Every unit at once: the rotated phenotypes and the fits on `side`, beside the rotated variants and their operands.
int run_grouped(flmm_context* ctx, const flmm_units* q, const UnitBufs& b, cudaStream_t main, cudaStream_t side, Events& ev) {
    const int N = q->N, Neff = N - q->D, P = q->P, U = q->n_units, R = b.R;
    const UnitBufs::Slot& s = b.slot[0];
    const int ldk = static_cast<int>(b.ldk);
    const bool pipe = side != main;
    auto after = [&](cudaEvent_t e, cudaStream_t first, cudaStream_t then) -> int {
        if (!pipe) return FLMM_OK;
        FLMM_CUDA(cudaEventRecord(e, first));
        FLMM_CUDA(cudaStreamWaitEvent(then, e, 0));
        return FLMM_OK;
    };
    std::vector<UnitTiles> us(U), f(U), w(U);
    std::vector<int> start(U + 1);
    int n_us = 0, n_f = 0, n_w = 0, big = 0, most = 0;
    auto tiles = [](int a, int rows_b) {
        return ((a + kUnitTileA - 1) / kUnitTileA) * ((rows_b + kUnitTileB - 1) / kUnitTileB);
    };
    for (int u = 0; u < U; ++u) {
        const int m0 = static_cast<int>(q->unit_start[u]), m = q->unit_count[u];
        start[u] = m0;
        start[u + 1] = m0 + m;
        us[u] = {n_us, m0, m, u * ldk, Neff};
        f[u] = {n_f, m0, m, u * R, R};
        w[u] = {n_w, u * P, P, m0, m};
        n_us += tiles(m, Neff);
        n_f += tiles(m, R);
        n_w += tiles(P, m);
        if (m > most) {
            most = m;
            big = u;
        }
    }
    const int M = start[U];
    int rc;
    if ((rc = put(us.data(), U, b.tiles_us, main)) || (rc = put(f.data(), U, b.tiles_f, main)) ||
        (rc = put(w.data(), U, b.tiles_w, main)) || (rc = put(start.data(), U + 1, b.start, main)))
        return rc;
    // every unit's eigenvector rows from a multiple of ldk on, zeros between
    const size_t pad = ldk - Neff, row = sizeof(__half) * s.Us.ld;
    if (pad) {
        for (__half* h : {s.Us.hi, s.Us.lo})
            FLMM_CUDA(cudaMemset2DAsync(h + Neff * s.Us.ld, ldk * row, 0, pad * row, U, main));
        FLMM_CUDA(cudaMemset2DAsync(s.Us.scale + Neff, ldk * sizeof(float), 0, pad * sizeof(float), U, main));
    }
    if ((rc = split_units(q->U + static_cast<int64_t>(q->D) * N, N, static_cast<int64_t>(N) * N, Neff, N, U, s.Us.hi, s.Us.lo,
                          s.Us.ld, ldk, s.Us.scale, main)))
        return rc;
    if ((rc = after(ev.e[0], main, side))) return rc;
    if (P > 0) {
        const int64_t ldu = static_cast<int64_t>(U) * ldk;
        if ((rc = flmm_gemm_split_f16(ctx, q->Yh, q->Yl, q->Yscale, q->ldY, P, s.Us.hi, s.Us.lo, s.Us.scale, s.Us.ld,
                                      U * ldk, N, s.UY, ldu, 0, side)))
            return rc;
        if ((rc = fit_delta_units(b.s, Neff, s.UY, ldu, ldk, P, U, q->opts.n_grid, q->opts.log_delta_min,
                                  q->opts.log_delta_max, q->opts.refine, q->log_delta, s.idx, s.fit, side)))
            return rc;
        if ((rc = prep_columns_units(b.s32, Neff, s.UY, ldu, ldk, q->log_delta, P, U, b.shat, b.x0, kInterpH, R, b.A1h, b.A1l,
                                     b.ldk, b.Lh, b.Ll, b.ldr, b.sa1, b.sl, b.rWr, b.rWr0, side)))
            return rc;
    }
    if (M > 0) {
        if ((rc = gemm_units(ctx, q->Zh, q->Zl, q->Zscale, q->ldZ, M, s.Us.hi, s.Us.lo, s.Us.scale, s.Us.ld, U * ldk, N, b.US,
                             b.ldk, b.tiles_us, U, n_us, main)))
            return rc;
        if ((rc = flmm_wald_split_prep_variants(b.US, b.ldk, M, Neff, b.B1h, b.B1l, b.B2h, b.B2l, b.ldk, b.sb1, b.sb2, main)))
            return rc;
        // node values of sWs~: F (M, R) = (US o US) W~^T, every variant with its unit's weights
        if ((rc = gemm_units(ctx, b.B2h, b.B2l, b.sb2, b.ldk, M, b.Ws.hi, b.Ws.lo, b.Ws.scale, b.ldk, U * R, Neff, b.F, b.ldr,
                             b.tiles_f, U, n_f, main)))
            return rc;
        if ((rc = flmm_split_rows_f16(b.F, 0, b.ldr, M, R, b.Fs.hi, b.Fs.lo, b.Fs.ld, b.Fs.scale, main))) return rc;
    }
    if ((rc = after(ev.e[1], side, main)) || M == 0 || P == 0) return rc;
    const bool refine = q->opts.f_refine > 0.0 && q->n_real > 0;
    WaldUnits x;
    x.A1h = b.A1h, x.A1l = b.A1l, x.lda = b.ldk, x.sa1 = b.sa1;
    x.Lh = b.Lh, x.Ll = b.Ll, x.ldl = b.ldr, x.sl = b.sl, x.rWr = b.rWr, x.rWr0 = b.rWr0;
    x.P = P, x.n_real = q->n_real, x.n_units = U;
    x.B1h = b.B1h, x.B1l = b.B1l, x.ldb = b.ldk, x.sb1 = b.sb1;
    x.Fh = b.Fs.hi, x.Fl = b.Fs.lo, x.ldf = b.Fs.ld, x.sf = b.Fs.scale;
    x.M = M, x.Neff = Neff, x.R = R, x.rows = q->rows;
    x.f = q->f, x.beta = q->beta, x.se = q->se, x.sfve = q->sfve, x.ldo = q->ldo, x.max_F = q->max_F;
    x.f_refine = refine ? static_cast<float>(q->opts.f_refine) : INFINITY;
    x.flag_count = refine ? b.flag_count : nullptr;
    x.flags = refine ? b.flags : nullptr;
    x.flag_cap = refine ? b.cap : 0;
    if ((rc = wald_units(ctx, x, b.tiles_w, n_w, w[big], main))) return rc;
    if (refine && (rc = wald_refine_units(ctx, b.flags, b.flag_count, b.cap, x.f_refine, b.US, b.ldk, s.UY,
                                          static_cast<int64_t>(U) * ldk, ldk, b.s32, q->log_delta, P, Neff, M, q->n_real,
                                          b.start, U, q->rows, q->f, q->beta, q->se, q->sfve, q->ldo, q->max_F, main)))
        return rc;
    if (q->n_real == 0) return FLMM_OK;
    return fill_nullh2_units(q->log_delta, P, q->n_real, q->rows, b.start, U, most, q->nullh2, q->ldo, main);
}

}  // namespace

extern "C" int flmm_scan_units_workspace_bytes(const flmm_units* q, size_t* bytes) {
    FLMM_REQUIRE(bytes, "flmm_scan_units_workspace_bytes: bytes is NULL");
    int rc = check_units(q);
    if (rc) return rc;
    // enough for either form, whichever is configured when the scan runs
    *bytes = 0;
    for (const bool group : {false, true}) {
        Arena a(nullptr);
        UnitBufs b;
        if ((rc = carve_units(a, q, group, &b))) return rc;
        *bytes = std::max(*bytes, a.off + 2048);
    }
    return FLMM_OK;
}

extern "C" int flmm_scan_units(flmm_context* ctx, const flmm_units* q, void* work, size_t work_bytes, void* stream,
                               void* side_stream) {
    int rc = check_units(q);
    if (rc) return rc;
    FLMM_REQUIRE(ctx && work && q->U && q->evals && q->rows && q->max_F && q->log_delta &&
                     (q->P == 0 || (q->Yh && q->Yl && q->Yscale && q->ldY >= q->N)) && q->Zh && q->Zl && q->Zscale &&
                     q->ldZ >= q->N &&
                     (q->n_real == 0 || (q->f && q->beta && q->se && q->sfve && q->nullh2 && q->ldo >= q->n_real)),
                 "flmm_scan_units: operands or outputs missing");
    size_t need = 0;
    if ((rc = flmm_scan_units_workspace_bytes(q, &need))) return rc;
    if (work_bytes < need) return fail(FLMM_ERR_WORKSPACE, "flmm_scan_units: need %zu bytes, got %zu", need, work_bytes);
    Arena a(work);
    UnitBufs b;
    if ((rc = carve_units(a, q, units_pair_ok(), &b))) return rc;
    const int Neff = q->N - q->D, U = q->n_units;
    cudaStream_t main = as_stream(stream), side = as_stream(side_stream);
    Events ev;
    if ((rc = ev.make())) return rc;
    // everything that the spectra decide, for all units
    k_unit_spectra<<<dim3(ceil_div(Neff, 256), U), 256, 0, main>>>(q->evals, q->N, q->D, b.s, b.s32);
    if ((rc = check_launch("k_unit_spectra"))) return rc;
    if ((rc = interp_units(b.s, Neff, U, b.shat, b.x0, kInterpH, b.R, b.W, main))) return rc;
    if ((rc = flmm_split_rows_f16(b.W, 1, Neff, U * b.R, Neff, b.Ws.hi, b.Ws.lo, b.ldk, b.Ws.scale, main))) return rc;
    const bool pipe = side != main;
    if (b.grouped) {
        try {
            rc = run_grouped(ctx, q, b, main, side, ev);
        } catch (const std::bad_alloc&) {  // (its tables; before anything is launched)
            rc = fail(FLMM_ERR_ARG, "flmm_scan_units: out of host memory");
        }
        if (rc && pipe && cudaEventRecord(ev.e[0], side) == cudaSuccess) cudaStreamWaitEvent(main, ev.e[0], 0);
        return rc;
    }
    auto record = [&](cudaEvent_t e, cudaStream_t s) { return !pipe || cudaEventRecord(e, s) == cudaSuccess; };
    auto wait = [&](cudaStream_t s, cudaEvent_t e) { return !pipe || cudaStreamWaitEvent(s, e, 0) == cudaSuccess; };
    // slot 0 and 1 alternate; e[1 + slot]: its column side is done, e[3 + slot]: its variant side is
    bool ok = record(ev.e[0], main) && wait(side, ev.e[0]);
    if (ok) rc = unit_columns(ctx, q, b, 0, side);
    ok = ok && record(ev.e[1], side);
    for (int u = 0; u < U && ok && !rc; ++u) {
        if (u + 1 < U) {
            if (u >= 1) ok = wait(side, ev.e[3 + ((u + 1) & 1)]);
            if (ok) rc = unit_columns(ctx, q, b, u + 1, side);
            ok = ok && record(ev.e[1 + ((u + 1) & 1)], side);
        }
        ok = ok && wait(main, ev.e[1 + (u & 1)]);
        if (ok && !rc) rc = unit_variants(ctx, q, b, u, main);
        ok = ok && record(ev.e[3 + (u & 1)], main);
    }
    // after an error the side stream may still be at work in the workspace: `stream` follows it before the caller does
    if (pipe && (rc || !ok) && cudaEventRecord(ev.e[0], side) == cudaSuccess) cudaStreamWaitEvent(main, ev.e[0], 0);
    if (!rc && !ok) return fail(FLMM_ERR_CUDA, "flmm_scan_units: %s", cudaGetErrorString(cudaGetLastError()));
    return rc;
}
