// The fast form's chromosome work issued from native code on caller-owned buffers: what fasterlmm_gb300.fast.scan_t runs.
//
//   flmm_loco_kinships_f32   per-chromosome Grams of a kinship panel (split-FP16 tensor-core products), the LOCO kinships
//                            of every unit and their projection off the covariates
//   flmm_scan_units          every unit's column side (eigenvector split, UY rotation, delta fit) and variant side (US
//                            rotation, Wald operands, fused Wald, strong-test re-evaluation, nullh2), the column side of
//                            unit u + 1 on a second stream beside the variant side of unit u
//
// Each unit is ~20 launches of a few microseconds for ordinary studies, and issuing them from Python cost 10-20 us each:
// 150 samples x 1,500 variants on 16 chromosomes took 10.2 ms in 505 launches, 4.35 here.  What depends on the spectra
// alone (mean, FP32 copies, sWs node weights and their split) and the projections run for all units in one launch each.
// The launches and their arithmetic are otherwise those of the C entry points called one by one.
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>
#include <cmath>

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
    UnitGram host[256];
    for (int u0 = 0; u0 < n_units; u0 += 256) {  // (pageable copies of a few hundred bytes are staged at once)
        const int n = std::min(256, n_units - u0);
        for (int u = 0; u < n; ++u) {
            const int b = unit_block[u0 + u];
            host[u] = UnitGram{b, static_cast<double>(M - (b >= 0 ? counts[b] : 0))};
        }
        FLMM_CUDA(cudaMemcpyAsync(units + u0, host, sizeof(UnitGram) * n, cudaMemcpyHostToDevice, st));
    }
    k_unit_kinships<<<dim3(ceil_div(nn, 256), n_units), 256, 0, st>>>(Gtot, grams, nn, units, Kp);
    if ((rc = check_launch("k_unit_kinships"))) return rc;
    return project_kinships(Kp, Qx, N, D, n_units, proj, st);
}

// ---- units ------------------------------------------------------------------------------------------------------

namespace {

struct UnitBufs {
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
    float* US;
    __half *A1h, *A1l, *Lh, *Ll, *B1h, *B1l, *B2h, *B2l;
    float *sa1, *sl, *rWr, *rWr0, *sb1, *sb2, *F;
    SplitBuf Fs;
    int32_t *flags, *flag_count;
    int R, cap;
    int64_t ldk, ldr;
    double x0;
};

int carve_units(Arena& a, const flmm_units* q, UnitBufs* b) {
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
    for (auto& s : b->slot) {
        s.Us = take_split(a, Neff, pad8(q->N));
        s.UY = a.of<float>(P * b->ldk);
        s.idx = a.of<int32_t>(P);
        s.fit = a.take(b->fit_bytes);
    }
    const size_t M = mc;
    b->US = a.of<float>(M * b->ldk);
    b->A1h = a.of<__half>(P * b->ldk);
    b->A1l = a.of<__half>(P * b->ldk);
    b->Lh = a.of<__half>(P * b->ldr);
    b->Ll = a.of<__half>(P * b->ldr);
    for (float** x : {&b->sa1, &b->sl, &b->rWr, &b->rWr0}) *x = a.of<float>(P);
    for (__half** x : {&b->B1h, &b->B1l, &b->B2h, &b->B2l}) *x = a.of<__half>(M * b->ldk);
    for (float** x : {&b->sb1, &b->sb2}) *x = a.of<float>(M);
    b->F = a.of<float>(M * b->ldr);
    b->Fs = take_split(a, mc, pad8(b->R));
    const int64_t tests = static_cast<int64_t>(mc) * q->n_real;
    b->cap = q->opts.f_refine > 0.0 ? static_cast<int>(std::min<int64_t>(tests, q->refine_cap)) : 0;
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
    FLMM_REQUIRE(q && q->N > q->D && q->D >= 1 && q->P >= 0 && q->n_real >= 0 && q->n_real <= q->P && q->n_units > 0 &&
                     q->unit_start && q->unit_count && q->opts.n_grid >= 1 && q->opts.log_delta_max > q->opts.log_delta_min &&
                     q->refine_cap >= 0,
                 "flmm_scan_units: bad arguments");
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

}  // namespace

extern "C" int flmm_scan_units_workspace_bytes(const flmm_units* q, size_t* bytes) {
    FLMM_REQUIRE(bytes, "flmm_scan_units_workspace_bytes: bytes is NULL");
    int rc = check_units(q);
    if (rc) return rc;
    Arena a(nullptr);
    UnitBufs b;
    if ((rc = carve_units(a, q, &b))) return rc;
    *bytes = a.off + 2048;
    return FLMM_OK;
}

extern "C" int flmm_scan_units(flmm_context* ctx, const flmm_units* q, void* work, size_t work_bytes, void* stream,
                               void* side_stream) {
    int rc = check_units(q);
    if (rc) return rc;
    FLMM_REQUIRE(ctx && work && q->U && q->evals && q->rows && q->max_F && q->log_delta &&
                     (q->P == 0 || (q->Yh && q->Yl && q->Yscale && q->ldY >= q->N)) && q->Zh && q->Zl && q->Zscale &&
                     q->ldZ >= q->N && (q->n_real == 0 || (q->f && q->beta && q->se && q->sfve && q->nullh2 && q->ldo >= q->n_real)),
                 "flmm_scan_units: operands or outputs missing");
    size_t need = 0;
    if ((rc = flmm_scan_units_workspace_bytes(q, &need))) return rc;
    if (work_bytes < need) return fail(FLMM_ERR_WORKSPACE, "flmm_scan_units: need %zu bytes, got %zu", need, work_bytes);
    Arena a(work);
    UnitBufs b;
    if ((rc = carve_units(a, q, &b))) return rc;
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
