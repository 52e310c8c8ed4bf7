// FP64 products on the FP16 tensor cores.
//
// GB300's FP64 pipe gives ~1.1 TFLOP/s, its FP16 tensor cores ~1,900, so a product C = A B^T of FP64 matrices is faster
// as several exact FP16 products.  Method: the error-free splitting of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms
// 59, 2012) on tensor cores as in Mukunoki, Ozaki, Ogita and Imamura (ISC 2020), with the level sums kept as integers.
// Every row is rounded once to 55 bits below its leading bit and written as eight balanced digits,
//     x = 2^(e - 6) (d_0 + d_1 2^-7 + ... + d_7 2^-49),  -64 <= d_t <= 64,
// e the binary exponent of the row's largest |x|.  Digits are exact in FP16; products of two digits are integers of at
// most 12 bits.  Plane pairs (i, j) of equal level l = i + j share one FP32 accumulator in tensor memory; levels 0..7
// are kept (36 pairs).  A level holds at most eight pairs, so its sum over a chunk of 512 terms is at most
// 8 * 512 * 2^12 = 2^24 in magnitude: every accumulation is exact.  The epilogue converts the level sums to integers
// and adds them into two 64-bit integers per output (levels 0..3 and 4..7), exactly, over all chunks, and rounds once:
//     C = 2^(e_a + e_b - 61) (2^28 hi + lo).
// What is lost is the rounding to 55 bits and the levels from 8 on (weight 2^-56 against the row maxima): fixed-point
// operands, whose entries far below their row's largest hold fewer bits than FP64's.  For rows whose largest entry is a few
// times their usual one this is smaller than the rounding of an FP64 sum of K terms (at K = 800 a scan's sums are 0.1 to 0.4
// of it off, at K = 100 0.3 to 0.9; measured against exact sums in tests/test_gpu_oz64.py).  The loss grows with the spread
// of both rows (after balancing, oz_balance), so every tile of rows carries its largest ratio; a tile pair whose product of
// ratios exceeds quality_limit, and any row that is not finite or whose exponent is out of range, is left to k_marked_f64,
// which forms those tiles on the FP64 pipe; and all of them where k_oz64 gave up a bounded wait, so that its callers need
// not wait for the device to see whether it did.
//
// Kernel: persistent CTA pairs; tiles of 256 A rows (128 a CTA) x 64 B rows, 8 levels x 64 columns = all of tensor memory.
// Warp 0 of each CTA issues its TMA loads: a stage is 16 deep, 8 x 4 KB of its own A rows and 8 x 1 KB of half the B rows =
// 40 KB in four boxes of 128-byte rows that hold four planes each, four stages.  Warp 1 of the even CTA issues the 36 MMAs
// of a stage (M = 256, N = 64, K = 16 over both), warps 2..17 drain the levels; tensor memory is handed back before the
// outputs are rounded and stored, so only the drain itself (8 x 64 columns per 512 terms, 4,300 cycles) interrupts the
// MMAs.  A pair's MMA reads 5 KB of operands a CTA where a CTA by itself reads 6 for half the work; and see elect_one: with
// an MMA's operands moved to uniform registers one by one, neither form went below 73 cycles an MMA.  Both products of 660
// columns x 4,000 variants x 800 samples with 5 covariates: 1.19 -> 0.78 ms (pairs by themselves 1.24).
#include <cuda.h>
#include <math.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "flmm_oz64.cuh"
#include "flmm_tc.cuh"

using namespace flmm;
using namespace flmm::tc;

namespace {

constexpr int kLevels = 8;
constexpr int kChunk = 512;  // terms of one exact accumulation
constexpr int kBK = 16;      // depth of one stage: a row's eight planes of 16 elements are 256 bytes, two 128-byte boxes
constexpr int kRowElems = kOzPlanes * kBK;            // elements of a row in one stage
constexpr int kABox = kOzRowsA * 128, kBBox = kOzRowsB / 2 * 128;
constexpr int kStageBytes = 2 * (kABox + kBBox);
constexpr int kStages = 4;
constexpr uint32_t kSBO = 1024;     // bytes between 8-row groups
constexpr uint32_t kSwizzle128 = 2u;
constexpr int kTmemCols = kLevels * kOzRowsB;
constexpr int kEpiWarps = 16;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kEpiCols = kOzRowsB / (kEpiWarps / 4);  // output columns per epilogue thread
constexpr int kOutCols = 8;                           // outputs of a row that pass through shared memory together
constexpr int kOutBytes = 32 * (kOutCols + 1) * 8;    // of a warp
constexpr int kSmemBytes = kStages * kStageBytes + kEpiWarps * kOutBytes + 256 + 1024;
constexpr int kMaxExp = 450;  // |e| beyond this: the scale 2^(e_a + e_b - 61) could leave FP64's range
static_assert(kTmemCols == 512 && kSmemBytes <= 227 * 1024 && kEpiCols == 16, "budgets");

// Largest product of two tiles' qualities that the digits take.  The loss of a sum is ~2^-56 sqrt(K) of the product of the
// row maxima.
//   kPlain (max/rms): an FP64 sum of terms of either sign is off by ~2^-53 K / 5 of the rms product, so the line goes with
//   sqrt(K).  Measured on a scan's operands at K = 1,000, relative to the row norms: ratios 10 x 5 leave 1.1e-17 where the
//   FP64 sum leaves 3.9e-17, so the two meet near a product of 150.
//   kBalanced (max/mean, which unlike max/rms keeps growing when one entry dominates a row: balancing can put a row's
//   largest entry where the other row is small, and max/rms of such a row is sqrt(K) at most).  A scan's tiles have products
//   of up to 7 sqrt(K) at K = 100 and 4 sqrt(K) at K = 1,000, and are 0.9 and 0.35 of the FP64 sum off; a row with one
//   dominating entry has 4 K.  At the line the digits lose 2 to 3 times what the FP64 sum does where one entry is large, and
//   8 times at worst, where the other row's entry is as small as that one is large (both of 5e-17 of the norms).  A sum of
//   non-negative terms is off by 2^-53 K^1.5 / 6 of the product of means: a scan's tiles have products of up to 0.9 K (K =
//   100) and 0.15 K (K = 1,000), and the two meet near 0.7 K.
//   kTerms: with A over sqrt(mean w) the loss of a term is 2^-56 of the product against sqrt(sum w b^2), twice that of the
//   term's square against sum w b^2, whose own FP64 sum is off by 2^-53 sqrt(K) / 6.
__host__ inline float quality_limit(OzGate gate, bool square, int K) {
    const float k = static_cast<float>(K), root = sqrtf(k);
    if (gate == OzGate::kPlain) return 4.0f * root;
    if (gate == OzGate::kTerms) return 0.7f * root;
    return square ? k : 8.0f * root;
}

struct OzMaps {
    CUtensorMap a, b;
};

struct OzArgs {
    int Ma, Nb, K, batches;
    int tiles_i, tiles_m;  // of 128 A rows, of 64 B rows
    int pairs_i;           // of 256 A rows
    const int* ea;
    const int* eb;
    const float* qa;
    const float* qb;
    float limit[2];  // per batch
    double* C;
    int64_t ldc, c_stride;
    const double* D;
    int64_t ldd;
    int* err;
};

// ---- digits ---------------------------------------------------------------------------------------------------

constexpr int kMaxBalance = 150;  // |e_k| used at most

// most[g][k] = largest high word of the finite |X[., k]| over the rows of group g (k_balance), then the exponent of the
// groups' median (k_balance_exp).  A block reads 32 columns of a group.
__global__ void __launch_bounds__(256)
k_balance(const double* __restrict__ X, int64_t ldx, int rows, int K, int* __restrict__ most) {
    __shared__ int red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane, g = blockIdx.y;
    const int r1 = static_cast<int>(static_cast<int64_t>(rows) * (g + 1) / gridDim.y);
    int m = 0;
    if (k < K) {
        const int* x = reinterpret_cast<const int*>(X) + 1;  // high words
#pragma unroll 8
        for (int r = static_cast<int>(static_cast<int64_t>(rows) * g / gridDim.y) + warp; r < r1; r += 8) {
            const int h = x[2 * (r * ldx + k)] & 0x7fffffff;
            m = h < 0x7ff00000 ? max(m, h) : m;
        }
    }
    red[warp][lane] = m;
    __syncthreads();
    if (warp == 0 && k < K) {
        for (int w = 1; w < 8; ++w) m = max(m, red[w][lane]);
        most[static_cast<int64_t>(g) * K + k] = m;
    }
}

__global__ void k_balance_exp(const int* __restrict__ most, int groups, int* __restrict__ bal, int K) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    int x[kOzBalanceGroups];
#pragma unroll
    for (int g = 0; g < kOzBalanceGroups; ++g) x[g] = g < groups ? most[static_cast<int64_t>(g) * K + k] : 0x7fffffff;
    int mid = 0;
#pragma unroll
    for (int g = 0; g < kOzBalanceGroups; ++g) {
        int below = 0;  // groups before this one in order
#pragma unroll
        for (int h = 0; h < kOzBalanceGroups; ++h) below += x[h] < x[g] || (x[h] == x[g] && h < g);
        if (below == (groups - 1) / 2) mid = x[g];
    }
    bal[k] = max(-kMaxBalance, min(kMaxBalance, (mid >> 20) - 1023));
}

// One warp per row.  Pass 1: the row's largest |x 2^c| (c = times bal_k) as its bit pattern (integer maximum); pass 2: the
// 55-bit integer of every element, its digits by integer shifts, packed two elements to a word (1536 + d is exact in FP16
// with unit spacing, so subtracting 1536 leaves the digit).  16 bytes written per 8 read: bandwidth-bound.
template <bool SQ>
__global__ void __launch_bounds__(256)
k_digits64(const double* __restrict__ X, int64_t ldx, int rows, int K, const int* __restrict__ bal, int times,
           __half* __restrict__ planes, int64_t ldp, int* __restrict__ expo, float* __restrict__ mean,
           float* __restrict__ qual, int tile_rows, const int* __restrict__ w_expo, const float* __restrict__ w_mean, int per) {
    const int lane = threadIdx.x & 31;
    const int64_t j = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
    if (j >= rows) return;
    const double* x = X + j * ldx;
    constexpr unsigned long long kInf = 0x7ff0000000000000ull;
    unsigned long long mb = 0;
    for (int n = lane; n < K; n += 32) {
        double v = x[n];
        if (SQ) v = mul_rn(v, v);
        unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffull;
        const int eb = static_cast<int>(b >> 52) + (bal ? times * bal[n] : 0);  // biased exponent of x 2^c
        if (b >= kInf || eb >= 0x7ff) b = kInf;
        else if (eb > 0 && b >> 52) b = (b & 0xfffffffffffffull) | (static_cast<unsigned long long>(eb) << 52);
        else b = b != 0;  // denormal: below every usable exponent, above zero
        mb = b > mb ? b : mb;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, mb, o);
        mb = b > mb ? b : mb;
    }
    const int e = mb == 0 ? 0 : static_cast<int>(mb >> 52) - 1022;  // max = f 2^e, f in [0.5, 1)
    const bool bad = e > kMaxExp || e < -kMaxExp;                   // includes infinities, NaN and denormals
    __half* out = planes + j * ldp;
    float ss = 0.0f, sa = 0.0f;
    for (int n = 2 * lane; n < (K + kBK - 1) / kBK * kBK; n += 64) {
        long long v[2] = {0, 0};
        if (!bad) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (n + h >= K) continue;
                double y = x[n + h];
                if (SQ) y = mul_rn(y, y);
                const int up = 1023 + 55 - e + (bal ? times * bal[n + h] : 0);
                v[h] = __double2ll_rn(y * __longlong_as_double(static_cast<long long>(up) << 52));
                const float t = static_cast<float>(static_cast<int>(v[h] >> 32)) * 0x1p-23f;
                ss = fmaf(t, t, ss);
                sa += fabsf(t);
            }
        }
#pragma unroll
        for (int t = kOzPlanes - 1; t >= 0; --t) {
            int d[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (t > 0) {
                    d[h] = static_cast<int>((static_cast<unsigned>(v[h]) + 64u) & 127u) - 64;
                    v[h] = (v[h] - d[h]) >> 7;
                } else {
                    d[h] = static_cast<int>(v[h]);
                }
            }
            const unsigned word = (static_cast<unsigned>(0x6600 + d[1]) << 16) | static_cast<unsigned>(0x6600 + d[0]);
            const __half2 p = __hsub2(*reinterpret_cast<const __half2*>(&word), __half2half2(__ushort_as_half(0x6600)));
            *reinterpret_cast<__half2*>(out + (n / kBK) * kRowElems + t * kBK + n % kBK) = p;
        }
    }
    ss = warp_sum(ss);
    sa = warp_sum(sa);
    if (lane == 0) {
        expo[j] = bad ? 0 : e;
        const float n = static_cast<float>(K), m = sa / n;
        mean[j] = m;
        const float top = static_cast<float>(__longlong_as_double((mb & 0xfffffffffffffull) | (1022ull << 52)));  // over 2^e
        float q;
        if (mb == 0) q = 1.0f;  // zeros
        else if (w_expo != nullptr) {
            const int ew = w_expo[j / per];
            q = ldexpf(top * rsqrtf(ldexpf(w_mean[j / per], ew & 1)), e - (ew >> 1));
        }
        else q = bal != nullptr ? top / m : top * sqrtf(n / ss);
        q = !bad && q < INFINITY ? fmaxf(w_expo != nullptr ? 0.0f : 1.0f, q) : INFINITY;
        atomicMax(reinterpret_cast<int*>(qual) + j / tile_rows, __float_as_int(q));
    }
}

__global__ void k_zero_f32(float* __restrict__ x, int n, int* __restrict__ flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = 0.0f;
    if (i < 2 && flag) flag[i] = 0;
}

// ---- the product ------------------------------------------------------------------------------------------------

// Tile t of the schedule: groups of at most kGroup pairs of A blocks, inside a group the pair fastest, so that the ~76
// tiles in flight share few A and B blocks in L2.
constexpr int kGroup = 6;

struct Tile {
    int b, ti, tm;  // ti: of 256 A rows in the schedule, of 128 for a CTA
};

__device__ __forceinline__ Tile tile_at(int t, int tiles_i, int tiles_m) {
    const int per = tiles_i * tiles_m;
    Tile r;
    r.b = t / per;
    int rem = t - r.b * per;
    const int g = rem / (kGroup * tiles_m);
    rem -= g * kGroup * tiles_m;
    const int gi = min(kGroup, tiles_i - g * kGroup);
    r.tm = rem / gi;
    r.ti = g * kGroup + rem - r.tm * gi;
    return r;
}

__device__ __forceinline__ bool tile_good(const OzArgs& a, const Tile& t) {
    // (an infinite quality makes the product infinite, or NaN with a zero one: neither is within the limit)
    return t.ti < a.tiles_i && a.qa[t.b * a.tiles_i + t.ti] * a.qb[t.b * a.tiles_m + t.tm] <= a.limit[t.b];
}

// The pair's tile: formed if either half is good (digits of rows that are not finite are zeros).
__device__ __forceinline__ bool pair_good(const OzArgs& a, const Tile& t) {
    return tile_good(a, Tile{t.b, 2 * t.ti, t.tm}) || tile_good(a, Tile{t.b, 2 * t.ti + 1, t.tm});
}

// Descriptors differ in their low words only (the tile's address in 16-byte units): plane t lies in box t / 4, 32 bytes
// further along its rows per plane.
__device__ __forceinline__ uint64_t plane_desc(uint32_t lo, uint32_t hi) {
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

template <int I, int J>
__device__ __forceinline__ void mma_pair(uint32_t elected, uint32_t tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi,
                                         uint32_t acc0, uint32_t idesc) {
    mma_f16_pair(elected, tmem + static_cast<uint32_t>((I + J) * kOzRowsB),
            plane_desc(a_lo + (I / 4) * (kABox / 16) + 2 * (I % 4), hi),
            plane_desc(b_lo + (J / 4) * (kBBox / 16) + 2 * (J % 4), hi), idesc, I == 0 ? acc0 : 1u);
    if constexpr (J < kLevels - 1 - I) mma_pair<I, J + 1>(elected, tmem, a_lo, b_lo, hi, acc0, idesc);
    else if constexpr (I < kOzPlanes - 1) mma_pair<I + 1, 0>(elected, tmem, a_lo, b_lo, hi, acc0, idesc);
}

__global__ void __launch_bounds__(kThreads, 1) k_oz64(const __grid_constant__ OzMaps maps, const OzArgs args) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
    uint64_t* full = bars;                  // [kStages], used in the even CTA
    uint64_t* empty = bars + kStages;       // [kStages]
    uint64_t* acc_full = empty + kStages;   // chunk accumulated (MMA -> epilogue)
    uint64_t* acc_empty = acc_full + 1;     // chunk drained (both epilogues -> MMA), used in the even CTA
    uint64_t* final_bar = acc_empty + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(final_bar + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int cl = static_cast<int>(cluster_id_x()), n_cl = static_cast<int>(cluster_count_x());
    const int n_tiles = args.batches * args.pairs_i * args.tiles_m;
    const int n_kb = (args.K + kBK - 1) / kBK;
    constexpr int kChunkKb = kChunk / kBK;
    constexpr uint32_t idesc = idesc_f16_f32(2 * kOzRowsA, kOzRowsB);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2 * kEpiWarps);
        mbar_init(final_bar, 1);
        fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, kTmemCols);
        tmem_relinquish_pair();
    }
    fence_before_sync();
    __syncwarp();
    cluster_sync();  // barriers initialised and tensor memory allocated in both CTAs
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t full0 = map_to_rank(smem_u32(full), 0);
            int stage = 0;
            uint32_t phase = 0;
            bool armed[kStages] = {};
            uint32_t armed_phase[kStages] = {};
            bool ok = true;
            for (int t = cl; t < n_tiles && ok; t += n_cl) {
                const Tile tl = tile_at(t, args.pairs_i, args.tiles_m);
                if (!pair_good(args, tl)) continue;
                const int ya = tl.b * args.Ma + (2 * tl.ti + static_cast<int>(rank)) * kOzRowsA;
                const int yb = tl.b * args.Nb + tl.tm * kOzRowsB + static_cast<int>(rank) * (kOzRowsB / 2);
                for (int kb = 0; kb < n_kb; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1u, args.err, 21)) { ok = false; break; }
                    if (leader) {
                        mbar_arrive_expect_tx(&full[stage], 2 * kStageBytes);
                        armed[stage] = true;
                        armed_phase[stage] = phase;
                    }
                    const uint32_t bar = full0 + static_cast<uint32_t>(stage * 8);
                    uint8_t* base = smem + stage * kStageBytes;
                    const int x = kb * kRowElems;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        tma_load_2d_pair(base + h * kABox, &maps.a, x + h * (kRowElems / 2), ya, bar);
                        tma_load_2d_pair(base + 2 * kABox + h * kBBox, &maps.b, x + h * (kRowElems / 2), yb, bar);
                    }
                    if (++stage == kStages) { stage = 0; phase ^= 1u; }
                }
            }
            if (leader) {
                // the pair's copies of every armed phase have landed before the CTAs leave
                for (int s = 0; s < kStages; ++s)
                    if (armed[s]) mbar_drain(&full[s], armed_phase[s]);
            } else if (*reinterpret_cast<volatile int*>(args.err) != 0) {
                // the even CTA may have stopped waiting on this CTA's last copies: give them time to land
                for (int i = 0; i < 100; ++i) __nanosleep(1000);
            }
        }
    } else if (warp == 1) {
        if (leader) {
            const uint32_t elected = elect_one();
            int stage = 0;
            uint32_t phase = 0, tphase = 0;
            bool ok = true;
            for (int t = cl; t < n_tiles && ok; t += n_cl) {
                if (!pair_good(args, tile_at(t, args.pairs_i, args.tiles_m))) continue;
                for (int kb = 0; kb < n_kb && ok; ++kb) {
                    const bool first = kb % kChunkKb == 0;
                    if (first) {
                        if (!mbar_wait_cluster_warp(acc_empty, tphase ^ 1u, args.err, 22)) { ok = false; break; }
                        fence_after_sync();
                    }
                    if (!mbar_wait_warp(&full[stage], phase, args.err, 23)) { ok = false; break; }
                    fence_after_sync();
                    const uint64_t d0 = smem_desc(smem_u32(smem + stage * kStageBytes), kSBO, kSwizzle128);
                    const uint32_t lo = static_cast<uint32_t>(d0);
                    mma_pair<0, 0>(elected, tmem_base, lo, lo + 2 * (kABox / 16), static_cast<uint32_t>(d0 >> 32),
                                   first ? 0u : 1u, idesc);
                    if (elected) mma_commit_pair(&empty[stage], 3);
                    if (++stage == kStages) { stage = 0; phase ^= 1u; }
                    if ((kb + 1) % kChunkKb == 0 || kb + 1 == n_kb) {
                        if (elected) mma_commit_pair(acc_full, 3);
                        tphase ^= 1u;
                    }
                }
            }
            if (elected) mma_commit_pair(final_bar, 3);
            mbar_drain(final_bar, 0);
        } else if (lane == 0) {
            // odd CTA: its shared and tensor memory stay live until the even CTA's last MMA has completed
            mbar_drain(final_bar, 0);
        }
    } else {
        // warp w reads TMEM lanes 32 (w % 4) .. +31 (thread = one A row) and columns 16 ((w - 2) / 4) .. +15 of every
        // level
        const int q = warp & 3;
        const int c0 = ((warp - 2) >> 2) * kEpiCols;
        const uint32_t tl0 = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(c0);
        const uint32_t acc_empty0 = map_to_rank(smem_u32(acc_empty), 0);
        double* buf = reinterpret_cast<double*>(smem + kStages * kStageBytes + 256 + (warp - 2) * kOutBytes);
        uint32_t tphase = 0;
        bool ok = true;
        for (int t = cl; t < n_tiles && ok; t += n_cl) {
            const Tile tl = tile_at(t, args.pairs_i, args.tiles_m);
            const Tile half{tl.b, 2 * tl.ti + static_cast<int>(rank), tl.tm};
            const bool good = tile_good(args, half);
            if (warp == 2 && lane == 0 && !good && half.ti < args.tiles_i) args.err[1] = 1;  // k_marked_f64 has work
            if (!pair_good(args, tl)) continue;
            long long hi[kEpiCols], lo[kEpiCols];
#pragma unroll
            for (int c = 0; c < kEpiCols; ++c) hi[c] = lo[c] = 0;
            for (int kb = 0; kb < n_kb; kb += kChunkKb) {
                const bool got = mbar_wait(acc_full, tphase, args.err, 24);
                if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
                fence_after_sync();
                float v[kEpiCols];
#pragma unroll
                for (int l = 0; l < kLevels / 2; ++l) {
                    tmem_ld16_wait(tl0 + static_cast<uint32_t>(l * kOzRowsB), v);
#pragma unroll
                    for (int c = 0; c < kEpiCols; ++c)
                        hi[c] += static_cast<long long>(__float2int_rn(v[c])) * (1 << (7 * (kLevels / 2 - 1 - l)));
                }
#pragma unroll
                for (int l = kLevels / 2; l < kLevels; ++l) {
                    tmem_ld16_wait(tl0 + static_cast<uint32_t>(l * kOzRowsB), v);
#pragma unroll
                    for (int c = 0; c < kEpiCols; ++c)
                        lo[c] += static_cast<long long>(__float2int_rn(v[c])) * (1 << (7 * (kLevels - 1 - l)));
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster_relaxed(acc_empty0);
                tphase ^= 1u;
            }
            if (!ok) break;
            if (!good) continue;
            // the outputs leave through shared memory, so that lanes go along the rows of C (and D)
            const int i0 = half.ti * kOzRowsA + q * 32;
            const int ea = i0 + lane < args.Ma ? args.ea[tl.b * args.Ma + i0 + lane] : 0;
            double* C = args.C + tl.b * args.c_stride;
#pragma unroll
            for (int h = 0; h < kEpiCols; h += kOutCols) {
                const int m0 = tl.tm * kOzRowsB + c0 + h;
                const int* eb = args.eb + tl.b * args.Nb + m0;
                __syncwarp();
#pragma unroll
                for (int c = 0; c < kOutCols; ++c) {
                    const int e = ea + (m0 + c < args.Nb ? eb[c] : 0);
                    const double s = __longlong_as_double(static_cast<long long>(1023 + e - 61) << 52);
                    buf[lane * (kOutCols + 1) + c] =
                        fma(static_cast<double>(hi[h + c]), 0x1p28, static_cast<double>(lo[h + c])) * s;
                }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < kOutCols; ++u) {
                    const int rr = (32 / kOutCols) * u + lane / kOutCols, c = lane % kOutCols;
                    if (i0 + rr < args.Ma && m0 + c < args.Nb) {
                        const double v = buf[rr * (kOutCols + 1) + c];
                        const int64_t i = i0 + rr;
                        C[i * args.ldc + m0 + c] = args.D ? args.D[i * args.ldd + m0 + c] - v : v;
                    }
                }
            }
        }
    }

    fence_before_sync();
    __syncwarp();
    cluster_sync();  // no CTA leaves while its peer may still signal its barriers or read its operands
    if (warp == 1) {
        fence_after_sync();
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

// ---- tiles left to the FP64 pipe ----------------------------------------------------------------------------------

constexpr int kST = 16, kSK = 16, kSThreads = 256;
constexpr int kSubs = (kOzRowsA / kST) * (kOzRowsB / kST);  // 16 x 16 outputs of a digit tile
constexpr int kNoPairs = 0x01010101;  // error word of a product that k_oz64 was not launched for

// The tiles of C whose digits are not good, or all after an error, in FP64: every block lists them in the same order and takes
// its share of their 16 x 16 parts, an output a thread.  One tile as two blocks of 64 x 64 outputs held up a launch for K
// 64^2 / 2 cycles of an SM's FP64 pipe (2,338 columns x 445 variants x 281 with one such tile: 0.22 of 0.62 ms).  Where D is C
// and k_oz64 gave up, some of D is gone: all NaN.
__global__ void __launch_bounds__(kSThreads)
k_marked_f64(const OzArgs args, const double* __restrict__ Xa, int64_t lda, int64_t xa_stride,
             const double* __restrict__ Xb, int64_t ldb, int square0, int square1) {
    __shared__ double As[kSK][kST + 1];
    __shared__ double Bs[kSK][kST + 1];
    __shared__ int list[kSThreads], before[kSThreads / 32 + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
    const int err = args.err[0];
    if (err == 0 && args.err[1] == 0) return;
    const bool lost = args.D == args.C && err != 0 && err != kNoPairs;
    const int per = args.tiles_i * args.tiles_m, total = args.batches * per;
    int64_t part = blockIdx.x;  // the block's next part, from the first of the tiles listed on
    for (int t0 = 0; t0 < total; t0 += kSThreads) {
        const int t = t0 + tid, in = t % per;
        const bool bad = t < total && (err != 0 || !tile_good(args, Tile{t / per, in / args.tiles_m, in % args.tiles_m}));
        const unsigned mask = __ballot_sync(0xffffffffu, bad);
        if (lane == 0) before[warp + 1] = __popc(mask);
        __syncthreads();
        if (tid == 0) {
            before[0] = 0;
            for (int w = 1; w <= kSThreads / 32; ++w) before[w] += before[w - 1];
        }
        __syncthreads();
        if (bad) list[before[warp] + __popc(mask & ((1u << lane) - 1u))] = t;
        const int parts = before[kSThreads / 32] * kSubs;
        __syncthreads();
        for (; part < parts; part += gridDim.x) {
            const int tile = list[part / kSubs], sub = static_cast<int>(part % kSubs), rem = tile % per, b = tile / per;
            const int i0 = rem / args.tiles_m * kOzRowsA + sub / (kOzRowsB / kST) * kST;
            const int j0 = rem % args.tiles_m * kOzRowsB + sub % (kOzRowsB / kST) * kST;
            if (i0 >= args.Ma || j0 >= args.Nb) continue;
            const bool sq = (b == 0 ? square0 : square1) != 0;
            const double* a = Xa + b * xa_stride + static_cast<int64_t>(i0 + ty) * lda;
            const double* x = Xb + static_cast<int64_t>(j0 + ty) * ldb;
            double acc = 0.0;
            for (int k0 = 0; k0 < args.K; k0 += kSK) {
                const bool kin = k0 + tx < args.K;
                As[tx][ty] = (kin && i0 + ty < args.Ma) ? a[k0 + tx] : 0.0;
                const double v = (kin && j0 + ty < args.Nb) ? x[k0 + tx] : 0.0;
                Bs[tx][ty] = sq ? mul_rn(v, v) : v;
                __syncthreads();
#pragma unroll
                for (int k = 0; k < kSK; ++k) acc = fma(As[k][ty], Bs[k][tx], acc);
                __syncthreads();
            }
            const int i = i0 + ty, j = j0 + tx;
            if (i < args.Ma && j < args.Nb) {
                const double v = args.D ? args.D[static_cast<int64_t>(i) * args.ldd + j] - acc : acc;
                args.C[b * args.c_stride + static_cast<int64_t>(i) * args.ldc + j] = lost ? NAN : v;
            }
        }
        part -= parts;
        __syncthreads();  // the list is read
    }
}

size_t align_up(size_t n) { return (n + 1023) / 1024 * 1024; }

}  // namespace

namespace flmm {

size_t oz_operand_bytes(int rows, int K, int batches, int tile_rows) {
    const size_t ldp = (static_cast<size_t>(K) + kBK - 1) / kBK * kRowElems, n = static_cast<size_t>(rows) * batches;
    const size_t tiles = static_cast<size_t>((rows + tile_rows - 1) / tile_rows) * batches;
    return align_up(sizeof(__half) * n * ldp) + align_up(sizeof(int) * n) + align_up(sizeof(float) * n) +
           align_up(sizeof(float) * (tiles + 2));
}

OzOperand oz_carve(void* base, int rows, int K, int batches, int tile_rows) {
    OzOperand op;
    op.ldp = (static_cast<int64_t>(K) + kBK - 1) / kBK * kRowElems;
    op.rows = rows;
    op.K = K;
    op.batches = batches;
    op.tile_rows = tile_rows;
    const size_t n = static_cast<size_t>(rows) * batches;
    char* p = static_cast<char*>(base);
    op.planes = reinterpret_cast<__half*>(p);
    p += align_up(sizeof(__half) * n * op.ldp);
    op.expo = reinterpret_cast<int*>(p);
    p += align_up(sizeof(int) * n);
    op.mean = reinterpret_cast<float*>(p);
    p += align_up(sizeof(float) * n);
    op.qual = reinterpret_cast<float*>(p);
    op.err = reinterpret_cast<int*>(op.qual + static_cast<size_t>(op.tiles()) * batches);
    return op;
}

int oz_balance(const double* X, int64_t ldx, int rows, int K, int* bal, cudaStream_t st) {
    const int groups = std::max(1, std::min(rows, kOzBalanceGroups));
    int* most = bal + K;
    k_balance<<<dim3(ceil_div(K, 32), groups), 256, 0, st>>>(X, ldx, rows, K, most);
    int rc = check_launch("k_balance");
    if (rc) return rc;
    k_balance_exp<<<ceil_div(K, 128), 128, 0, st>>>(most, groups, bal, K);
    return check_launch("k_balance_exp");
}

int oz_digits(const OzOperand& op, int b, const double* X, int64_t ldx, bool square, const int* bal, int times,
              cudaStream_t st, OzWeights weights) {
    if (op.rows == 0) return FLMM_OK;
    const int64_t off = static_cast<int64_t>(b) * op.rows;
    float* qual = op.qual + static_cast<int64_t>(b) * op.tiles();
    k_zero_f32<<<ceil_div(op.tiles(), 256), 256, 0, st>>>(qual, op.tiles(), b == 0 ? op.err : nullptr);
    int rc = check_launch("k_zero_f32");
    if (rc) return rc;
    const int64_t w_off = weights.op ? weights.op->rows : 0;  // (batch 1)
    auto* k = square ? k_digits64<true> : k_digits64<false>;
    k<<<ceil_div(static_cast<int64_t>(op.rows) * 32, 256), 256, 0, st>>>(
        X, ldx, op.rows, op.K, bal, times, op.planes + off * op.ldp, op.ldp, op.expo + off, op.mean + off, qual, op.tile_rows,
        weights.op ? weights.op->expo + w_off : nullptr, weights.op ? weights.op->mean + w_off : nullptr, weights.per);
    return check_launch("k_digits64");
}

int oz_gemm(const OzOperand& A, const OzOperand& B, const OzProduct& p, cudaStream_t st) {
    if (A.rows == 0 || B.rows == 0) return FLMM_OK;
    if (A.batches > 2 || B.batches > 2 || A.K != B.K) return fail(FLMM_ERR_ARG, "oz_gemm: operands differ");
    const int64_t ra = static_cast<int64_t>(A.rows) * A.batches, rb = static_cast<int64_t>(B.rows) * B.batches;
    if (ra > 0x7fffffffLL || rb > 0x7fffffffLL || A.ldp > 0x7fffffffLL)
        return fail(FLMM_ERR_ARG, "oz_gemm: too large for a TMA map");
    OzMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    int rc;
    const int w = static_cast<int>(A.ldp);
    if ((rc = tc::make_map_f16(&maps.a, A.planes, static_cast<int>(ra), w, A.ldp, kRowElems / 2, kOzRowsA))) return rc;
    if ((rc = tc::make_map_f16(&maps.b, B.planes, static_cast<int>(rb), w, B.ldp, kRowElems / 2, kOzRowsB / 2))) return rc;
    static PairCache cache;
    int pairs = 0;
    if (use_pair_kernels() && (rc = pair_count(k_oz64, kThreads, kSmemBytes, cache, &pairs))) return rc;
    OzArgs a{};
    a.err = A.err;
    a.Ma = A.rows;
    a.Nb = B.rows;
    a.K = A.K;
    a.batches = A.batches < B.batches ? A.batches : B.batches;
    a.tiles_i = A.tiles();
    a.tiles_m = B.tiles();
    a.pairs_i = (a.tiles_i + 1) / 2;
    a.ea = A.expo;
    a.eb = B.expo;
    a.qa = A.qual;
    a.qb = B.qual;
    for (int b = 0; b < 2; ++b) a.limit[b] = quality_limit(p.gate, p.square[b], A.K);
    a.C = p.C;
    a.ldc = p.ldc;
    a.c_stride = p.c_stride;
    a.D = p.D;
    a.ldd = p.ldd;
    const int64_t tiles = static_cast<int64_t>(a.batches) * a.pairs_i * a.tiles_m;
    pairs = static_cast<int>(std::min<int64_t>(tiles, pairs));
    if (pairs > 0) {
        if ((rc = launch_pairs(k_oz64, pairs, kThreads, kSmemBytes, st, maps, a))) return rc;
        if ((rc = check_launch("k_oz64"))) return rc;
    } else {
        FLMM_CUDA(cudaMemsetAsync(a.err, kNoPairs & 0xff, sizeof(int), st));
    }
    int sms = 0;
    if ((rc = sm_count(&sms))) return rc;
    // (two blocks an SM: eight take 3 us longer to find that there is nothing to do)
    const int64_t parts = static_cast<int64_t>(a.batches) * a.tiles_i * a.tiles_m * kSubs;
    const int grid = static_cast<int>(std::min<int64_t>(int64_t{2} * sms, parts));
    k_marked_f64<<<grid, kSThreads, 0, st>>>(a, p.Xa, p.lda, p.xa_stride, p.Xb, p.ldb, p.square[0], p.square[1]);
    return check_launch("k_marked_f64");
}

bool oz_worth(int64_t Mr, int64_t Nr, int64_t K) { return K >= 32 && Mr * Nr * K >= 20000000; }

}  // namespace flmm
