// Blackwell (sm_103a) tensor-core primitives in inline PTX: mbarriers with bounded waits, TMA 2-D tile loads,
// tensor-memory (TMEM) allocation, tcgen05.mma (kind::f16, FP32 accumulate in TMEM), tcgen05.commit and
// tcgen05.ld.  Shared-memory operand tiles are K-major with the TMA's 64-byte or 128-byte swizzle, which is the
// canonical layout the MMA's shared-memory descriptors describe.
#pragma once

#include <cuda.h>
#include <stdint.h>

#include <mutex>

#include "flmm_common.cuh"

namespace flmm {
namespace tc {

// Bound on every spin-wait, in SM clock cycles (~2 s at 2 GHz).  A wait that runs out records an error code in a
// global flag and returns false; the kernel then winds down instead of hanging the GPU.
constexpr long long kWaitCycles = 4000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier -------------------------------------------------------------------------------------------------

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ uint32_t mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}

// Wait for the phase of `bar` with the given parity to complete.  Bounded: gives up after kWaitCycles, or as soon
// as another role of the kernel has raised *err; on giving up it raises *err with `code` and returns false.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0) {
            if (*reinterpret_cast<volatile int*>(err) != 0) return false;
            if (clock64() - t0 > kWaitCycles) {
                atomicCAS(err, 0, code);
                return false;
            }
        }
    }
}

// ---- TMA ------------------------------------------------------------------------------------------------------

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// 2-D tile load: box at element coordinates (x = inner / K, y = row) into shared memory, completion counted on
// `bar` in bytes.  x must be a multiple of 8 FP16 elements (16 bytes); callers only use multiples of the box width.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// ---- tensor memory ----------------------------------------------------------------------------------------------

// whole-warp operations
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- MMA ------------------------------------------------------------------------------------------------------

// Instruction descriptor, kind::f16: D = FP32 (bits 4-5 = 1), A = B = FP16 (bits 7-9, 10-12 = 0), both K-major
// (bits 15, 16 = 0), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_f16_f32(int M, int N) {
    return (1u << 4) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// Shared-memory matrix descriptor for a K-major swizzled tile: start address >> 4 (bits 0-13), leading byte
// offset 16 B (unused for swizzled K-major, bits 16-29), stride byte offset between 8-row groups >> 4
// (bits 32-45), descriptor version 1 (bits 46-47), swizzle mode (bits 61-63: 2 = 128 B, 4 = 64 B).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t sbo_bytes, uint32_t swizzle_mode) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
    d |= static_cast<uint64_t>(1u) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1u) << 46;
    d |= static_cast<uint64_t>(swizzle_mode & 7u) << 61;
    return d;
}

// One lane of a converged warp.  The MMA warps run their loops as a whole and leave the instructions themselves to this
// lane: the loops are then uniform, and descriptors and addresses live in uniform registers.  Behind `if (lane == 0)` each of
// an MMA's operands was moved there for every MMA, ~73 cycles between one and the next, where M = 128 x N = 64 x 16 takes 48
// and a CTA pair's 256 x 128 x 16 takes 64.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}

// a converged warp's wait (mbar_wait in every lane): true if all lanes saw the phase complete
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* err, int code) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, err, code));
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by the elected lane of a converged warp.
__device__ __forceinline__ void mma_f16(uint32_t elected, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
        : "memory");
}

// Arrive on `bar` once every tcgen05 operation issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Two 16-column loads (e.g. the same columns of two accumulators) and the wait for both, in one asm statement so
// that no use of the destination registers can be scheduled before tcgen05.wait::ld.
__device__ __forceinline__ void tmem_ld16x2(uint32_t ta, uint32_t tb, float (&va)[16], float (&vb)[16]) {
    uint32_t a[16], b[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, "
        "[%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]),
          "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]), "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15]),
          "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7]),
          "=r"(b[8]), "=r"(b[9]), "=r"(b[10]), "=r"(b[11]), "=r"(b[12]), "=r"(b[13]), "=r"(b[14]), "=r"(b[15])
        : "r"(ta), "r"(tb)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        va[i] = __uint_as_float(a[i]);
        vb[i] = __uint_as_float(b[i]);
    }
}

// One 16-column load and its wait.
__device__ __forceinline__ void tmem_ld16_wait(uint32_t ta, float (&va)[16]) {
    uint32_t a[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]),
          "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]), "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15])
        : "r"(ta)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) va[i] = __uint_as_float(a[i]);
}

// ---- CTA pairs (tcgen05 cta_group::2) -------------------------------------------------------------------------
// A cluster of two CTAs runs one MMA of M = 256 rows: each CTA holds its 128 A rows and half of the B rows in its
// own shared memory at the same offsets, the even CTA issues the MMA, and each CTA's tensor memory receives its
// own 128 rows of the product.  Every tcgen05 instruction of such a kernel carries .cta_group::2.

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_id_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_count_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}

// all threads of both CTAs; orders each thread's earlier memory operations before the peer's later ones
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// shared::cluster address of the variable at shared::cta address `saddr` in the cluster's CTA `rank`
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}

// arrive on an mbarrier of either CTA of the cluster (cluster address from map_to_rank)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}

// The same arrive without release semantics: for handing a drained tensor-memory slot back to the MMA issuer, where
// the only accesses to order are the caller's tcgen05.ld of the slot, which tcgen05.wait::ld has completed and
// tcgen05.fence::before_thread_sync orders before the arrive; the release would also wait for the thread's global
// stores to become visible at cluster scope.
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t bar_cluster) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}

__device__ __forceinline__ uint32_t mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}

// mbar_wait for a barrier whose arrivals come from the peer CTA (acquire at cluster scope)
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* err, int code) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if ((it & 255u) == 0) {
            if (*reinterpret_cast<volatile int*>(err) != 0) return false;
            if (clock64() - t0 > kWaitCycles) {
                atomicCAS(err, 0, code);
                return false;
            }
        }
    }
}

// 2-D tile load into this CTA's shared memory whose completion is counted on an mbarrier of either CTA of the
// pair (cluster address); same x alignment rule as tma_load_2d
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
        "%3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar_cluster)
        : "memory");
}

// one warp of each CTA of the pair: the same columns in both CTAs' tensor memory
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// a converged warp's wait for a barrier whose arrivals come from the peer CTA
__device__ __forceinline__ bool mbar_wait_cluster_warp(uint64_t* bar, uint32_t parity, int* err, int code) {
    return __all_sync(0xffffffffu, mbar_wait_cluster(bar, parity, err, code));
}

// D (+)= A B^T over the pair, issued by the elected lane of a converged warp of the even CTA
__device__ __forceinline__ void mma_f16_pair(uint32_t elected, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(elected)
        : "memory");
}

// arrive on the mbarrier at the same offset in each CTA of `cta_mask` once the pair's MMAs issued so far completed
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar, uint16_t cta_mask) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"(cta_mask)
        : "memory");
}

// FP16 matrix (rows, K) with row pitch ld elements (a multiple of 8, base 16-byte aligned) -> tiled TMA map with box
// {BK, box_rows}, BK 32 (64-byte swizzle) or 64 (128-byte swizzle); rows and columns outside the matrix read as zero.
int make_map_f16(CUtensorMap* map, const void* base, int rows, int K, int64_t ld, int BK, int box_rows);

// CTA pairs of a kernel (one CTA per SM) that the current device runs at once, 0 if none fits; sets its shared-memory
// limit.  `cache` is the kernel's own, by device.
struct PairCache {
    std::mutex mu;
    int pairs[64] = {};
    bool known[64] = {};
};

template <typename Kernel>
int pair_count(Kernel* kernel, int threads, int smem_bytes, PairCache& cache, int* out) {
    int dev = 0, sm = 0, n = 0;
    FLMM_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(FLMM_ERR_ARG, "pair_count: device %d", dev);
    std::lock_guard<std::mutex> lock(cache.mu);
    // (per device context, so set on every call; the call is cheap)
    FLMM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    if (!cache.known[dev]) {
        FLMM_CUDA(cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(static_cast<unsigned>(sm & ~1));
        cfg.blockDim = dim3(static_cast<unsigned>(threads));
        cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        FLMM_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
        cache.pairs[dev] = n;
        cache.known[dev] = true;
    }
    *out = cache.pairs[dev];
    return FLMM_OK;
}

// `pairs` CTA pairs of a kernel
template <typename... Params, typename... Args>
int launch_pairs(void (*kernel)(Params...), int pairs, int threads, int smem_bytes, cudaStream_t st, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FLMM_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    return FLMM_OK;
}

// Bounded wait that ignores the kernel's error flag: used at teardown to drain TMA copies still in flight.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > kWaitCycles) return;
    }
}

}  // namespace tc
}  // namespace flmm
