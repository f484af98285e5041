// tcgen05 (5th-generation tensor core) and TMEM helpers for sm_100a, written
// as inline PTX.  Descriptor bit layouts follow the PTX ISA for tcgen05:
//   shared-memory matrix descriptor (64 bit): start address >> 4 [0,14),
//   leading-dimension byte offset >> 4 [16,30), stride-dimension byte offset
//   >> 4 [32,46), descriptor version 1 [46,48), base offset [49,52), layout
//   (swizzle) type [61,64) with 0 = none, 2 = 128B, 4 = 64B, 6 = 32B;
//   instruction descriptor for kind::f16 and kind::f8f6f4 (32 bit): D format
//   [4,6) (1 = F32), A format [7,10) and B format [10,13) (kind::f16: 0 = F16,
//   1 = BF16; kind::f8f6f4: 0 = E4M3, 1 = E5M2), A/B major [15], [16]
//   (0 = K-major), N >> 3 [17,23), M >> 4 [24,29).
#pragma once

#include <stdint.h>

#include "common.cuh"

namespace gatlas {
namespace tc {

#ifdef __CUDACC__

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// mbarrier wait of one thread, bounded in wall time (ns).  Returns false on
// timeout or when *abort becomes non-zero.
__device__ __forceinline__ bool wait_timed(uint64_t *bar, uint32_t parity, uint64_t limit_ns,
                                           volatile int *abort) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (abort && *abort) return false;
        if (globaltimer() - t0 > limit_ns) return false;
    }
}

// The same for a whole converged warp.  Each lane polls by itself and may give
// up by itself (its own clock, the abort flag), so the lanes agree before one
// of them acts on the answer: false where any lane gave up.  Without the vote
// some lanes would leave while others went on to warp-wide instructions
// (elect.sync, TMEM loads) that then never complete.
__device__ __forceinline__ bool wait_warp(uint64_t *bar, uint32_t parity, uint64_t limit_ns, volatile int *abort) {
    return __all_sync(0xffffffffu, wait_timed(bar, parity, limit_ns, abort));
}

// The same where each lane that gives up returns from the kernel: the syncs,
// barriers and shuffles of the others wait only for threads that have not exited.
// (For the TMA GEMV kernels, whose warps wait once per 2 to 4 KiB: a vote after each
// wait cost them 3 %.)
__device__ __forceinline__ bool wait_or_exit(uint64_t *bar, uint32_t parity, uint64_t limit_ns, volatile int *abort) {
    return wait_timed(bar, parity, limit_ns, abort);
}

enum Swizzle : uint32_t { kSwizzleNone = 0, kSwizzle128B = 2, kSwizzle64B = 4, kSwizzle32B = 6 };

// K-major operand descriptor: 8-row core-matrix groups `sbo_bytes` apart,
// rows of the swizzle width; the leading byte offset is unused for swizzled
// K-major layouts and set to 16 bytes.
__device__ __forceinline__ uint64_t smem_desc_kmajor(uint32_t smem_addr, uint32_t sbo_bytes, uint32_t swz) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)(1u) << 16;                            // LBO = 16 B (unused)
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;     // SBO
    d |= (uint64_t)1 << 46;                               // version
    d |= (uint64_t)(swz & 7u) << 61;                      // layout type
    return d;
}

__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
    return (1u << 4)                    // D = F32
           | (1u << 7)                  // A = BF16
           | (1u << 10)                 // B = BF16
           | ((uint32_t)(N >> 3) << 17) // N
           | ((uint32_t)(M >> 4) << 24);// M
}

// kind::f8f6f4 with A = B = E4M3 (format code 0) and an F32 accumulator.
__host__ __device__ constexpr uint32_t idesc_e4m3_f32(int M, int N) {
    return (1u << 4)                    // D = F32
           | (0u << 7)                  // A = E4M3
           | (0u << 10)                 // B = E4M3
           | ((uint32_t)(N >> 3) << 17) // N
           | ((uint32_t)(M >> 4) << 24);// M
}

__device__ __forceinline__ void tmem_alloc(uint32_t *smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
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

// True on one lane of a converged warp.  MMAs issued under it from code that
// the whole warp runs keep their descriptors in uniform registers; under
// `lane == 0` every operand is moved there first.
__device__ __forceinline__ bool elect_one() {
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(on));
    return on != 0;
}

// D[tmem] (+)= A[smem desc] * B[smem desc]^T, single CTA, kind::f16.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// D[tmem] (+)= A * B^T with 8-bit floating-point operands (K = 32 per instruction).
__device__ __forceinline__ void mma_f8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives once on the mbarrier when all previously issued tcgen05 async
// operations of this thread have completed.
__device__ __forceinline__ void commit_to(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp receives
// lane (base lane + i), columns [col, col + 32).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

// 32 lanes x 16 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15])
        : "r"(taddr));
}

// 32 lanes x 8 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---- CTA pairs (cta_group::2): a cluster of two CTAs sharing one MMA ----

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// shared::cluster address of the variable at shared::cta address `addr` in
// CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// Whole-cluster execution barrier (every thread of every CTA).  The aligned
// forms need converged warps, whatever the code before them branched on.
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// mbarrier wait with cluster-scope acquire (the barrier receives arrivals
// from the other CTA of the pair), bounded in wall time.
__device__ __forceinline__ bool try_wait_cluster(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_timed_cluster(uint64_t *bar, uint32_t parity, uint64_t limit_ns,
                                                   volatile int *abort) {
    if (try_wait_cluster(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    while (true) {
        if (try_wait_cluster(bar, parity)) return true;
        if (abort && *abort) return false;
        if (globaltimer() - t0 > limit_ns) return false;
    }
}

__device__ __forceinline__ bool wait_warp_cluster(uint64_t *bar, uint32_t parity, uint64_t limit_ns,
                                                  volatile int *abort) {
    return __all_sync(0xffffffffu, wait_timed_cluster(bar, parity, limit_ns, abort));
}

// Launches on one stream that overlap (programmatic dependent launch): the next
// one may start once every CTA of this one has said so or ended; it waits until
// this one has ended and its writes are visible.
__device__ __forceinline__ void let_next_launch_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_launch_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Arrive on an mbarrier of another CTA of the cluster (shared::cluster address).
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t *smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
                 "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// D (both CTAs' TMEM, M = 256 split by rows) (+)= A (128 rows in each CTA's
// shared memory at the same offset) * B^T (N/2 rows in each CTA).
__device__ __forceinline__ void mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_f8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives once on the mbarrier at shared::cluster address `bar` (this CTA's
// or the peer's) when the pair MMAs issued so far by this thread complete.
__device__ __forceinline__ void commit_pair_to(uint32_t bar_cluster_addr) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     bar_cluster_addr)
                 : "memory");
}

// 3-D tensor-map load into this CTA's shared memory whose completion counts
// on the mbarrier at shared::cluster address `bar` (the pair leader's).
__device__ __forceinline__ void tma_load_3d_pair(void *smem_dst, const void *tmap, int32_t x, int32_t y, int32_t z,
                                                 uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar_cluster_addr)
        : "memory");
}

// L2 eviction priorities for cache-hinted loads (createpolicy, whole range).
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

// tma_load_3d / tma_load_3d_pair with an L2 eviction priority.
__device__ __forceinline__ void tma_load_3d_hint(void *smem_dst, const void *tmap, int32_t x, int32_t y, int32_t z,
                                                 uint64_t *bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d_pair_hint(void *smem_dst, const void *tmap, int32_t x, int32_t y,
                                                      int32_t z, uint32_t bar_cluster_addr, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(smem_dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar_cluster_addr), "l"(policy)
        : "memory");
}

#endif  // __CUDACC__

}  // namespace tc
}  // namespace gatlas
