// Grouped tensor-core matmul: hundreds of instances of different shapes and
// layouts (C_i = alpha_i * op(A_i) op(B_i) + beta_i * C_i) in one persistent
// launch.
//
// No reference counterpart as one kernel: the reference batches only equal
// shapes (packedCalc, KernelMatmulBuffer.hpp:229-230) and otherwise runs one
// kernel per problem.  Design for B200:
//  1. pack pass (one launch for all instances): every FP32 operand is split
//     into BF16 pieces and written tile-major in the exact shared-memory
//     image the MMA descriptors read: A as [mt][kt][128 rows x 128 B], B as
//     [nt][kt][BN rows x 128 B], each tile 128-byte swizzled (16-byte chunk
//     c of row r stored at chunk c ^ (r & 7)), zero padded past M, N, K.
//     The contraction then streams every tile with one 1-D bulk copy: no
//     per-instance tensor maps.  The pack itself stages its source tiles
//     with 16-byte async copies through a 3-stage shared-memory ring;
//  2. contraction: one CTA per SM walks a statically balanced list of
//     output tiles (longest first, greedy onto the least-loaded CTA) across
//     instances.  Warp 0 streams tiles through the mbarrier ring, warp 1
//     issues tcgen05.mma (N = the instance's tile width), warps 2..9 promote
//     the TMEM segments into FP32 registers and write C, overlapping the
//     epilogue of one tile with the main loop of the next (two TMEM
//     accumulators).
// The tile width BN (64, 128 or 256) is chosen per instance, by default from
// a per-size-bucket table that the autotuner fills.
// Every wait is bounded; a timeout sets the device fault word, stops the
// pipeline, drains the copies in flight and frees TMEM.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <queue>
#include <vector>

#include "../common.cuh"
#include "../device_state.cuh"
#include "../tcgen05.cuh"
#include "gemm_engines.hpp"
#include "grouped.hpp"
#include "tc_modes.cuh"

namespace gatlas {
namespace grp {

using tcg::BM;
constexpr int kPackBK = 64;              // K elements per pack item
constexpr uint32_t kPackRowBytes = 128;   // one pack item's row of one BF16 piece
constexpr uint32_t kRowBytes = 128;       // one contraction K slice of one row (128-byte swizzle)
constexpr int kBK = kRowBytes / 2;        // BF16 elements per contraction K slice
constexpr int kSlicesPerItem = (int)(kPackRowBytes / kRowBytes);
constexpr uint32_t kATileBytes = BM * kRowBytes;
constexpr int kDrainWarps = 8;            // a multiple of 4: kDrainParts warps per TMEM lane quarter
// Roles are whole warpgroups: warps 0 and 1 produce and issue (2 and 3 idle),
// warps 4..11 drain.  The first group gives its registers to the drain, whose
// 128 sums, a chunk of C and the tile's record do not fit the 168 that 384
// threads start with: 128 x 40 + 256 x 232 = 384 x 168.
constexpr int kThreads = 32 * (4 + kDrainWarps);
constexpr int kIssueRegs = 40, kDrainRegs = 232;
static_assert(128 * kIssueRegs + 32 * kDrainWarps * kDrainRegs <= kThreads * 168, "register split");
constexpr int kDrainParts = kDrainWarps / 4;          // column parts of a tile per lane quarter
constexpr int kPartCols = 256 / kDrainParts;          // columns in a part of the widest tile
constexpr uint32_t kTmemCols = 512;       // two accumulators of up to 256 columns
constexpr uint64_t kWaitNs = 2000000000ull;
constexpr int kPackRows = 128;            // rows per pack item
constexpr uint32_t kEpiTileBytes = 32 * 32 * 4;
constexpr uint32_t kEpiBytes = kDrainWarps * kEpiTileBytes;
static_assert(kDrainWarps % 4 == 0 && kPartCols % 32 == 0, "drain layout");
// The grouped engine stages 128-byte K slices (its packed tiles carry the
// 128-byte swizzle): the ring holds two split3 slices of a 128 x 256 tile (96
// KiB each) or four BF16 ones, beside the drain's staging.  It promotes after the same K as the single-instance
// engine (all of K for one-product BF16, 256 for split3), issuing the same
// MMA sequence (16-deep K steps in order, the products of each in order), so
// that each instance's result is bit-identical to it.
// Ring layout: a stage holds every piece of a 128-row A tile and of BROWS
// rows of B (one K slice): all 256 rows of the widest tile on a single CTA,
// its 128-row half on each CTA of a pair.
template <int MODE, int BROWS>
struct GLayout {
    using MD = tcg::Mode<MODE>;
    static constexpr int BK = kRowBytes / MD::ELEM;
    static constexpr uint32_t SWIZZLE = kRowBytes == 128 ? tc::kSwizzle128B : tc::kSwizzle64B;
    static constexpr uint32_t SBO = 8 * kRowBytes;
    static constexpr int KSTEPS = kRowBytes / 32;
    static constexpr uint32_t A_TILE = BM * kRowBytes;
    static constexpr uint32_t B_TILE = BROWS * kRowBytes;
    static constexpr uint32_t STAGE_BYTES = MD::NP * (A_TILE + B_TILE);
    static constexpr int FIT = (int)((226 * 1024 - 1024 - kEpiBytes) / STAGE_BYTES);
    static constexpr int STAGES = FIT < 8 ? FIT : 8;
    static constexpr uint32_t EPI_OFFSET = STAGES * STAGE_BYTES;  // a 32 x 32 staging tile of C per drain warp
    static constexpr uint32_t SMEM_BYTES = EPI_OFFSET + kEpiBytes + 1024;  // + alignment slack
    static_assert(STAGES >= 2, "grouped pipeline depth");
};
template <int MODE, bool PAIR>
using GLayoutOf = GLayout<MODE, PAIR ? 128 : 256>;
constexpr int grouped_seg_kblocks(int mode) { return mode == 0 ? tcg::kSegAll : 256 / kBK; }

// Packed byte offset of 16-byte chunk c (0..7) of row `row` of pack item kb
// (K elements 64 kb .. 64 kb + 63) in an operand of kt items per row block of
// tr rows.  Each row block is a run of K slices, each slice tr rows of
// kRowBytes; 16-byte chunk j of row r sits at chunk j ^ (r & 7) (128-byte
// swizzle) or j ^ ((r >> 1) & 3) (64-byte swizzle), the layouts the MMA's
// shared-memory descriptors read.
// tr is a power of two (128 rows of A; 64, 128 or 256 of B): shifts, because a
// 64-bit division per store was half of the pack pass's instructions.
__device__ __forceinline__ int64_t packed_offset(int64_t row, int kb, int c, int tr, int kt) {
    constexpr int per = (int)(kRowBytes / 16);  // chunks per slice row
    const int s = kb * kSlicesPerItem + c / per, j = c % per;
    const int swz = kRowBytes == 128 ? (int)(row & 7) : (int)((row >> 1) & 3);
    const int shift = 31 - __clz(tr);
    return (((row >> shift) * (int64_t)(kt * kSlicesPerItem) + s) << shift) * kRowBytes +
           (row & (tr - 1)) * kRowBytes + ((j ^ swz) << 4);
}

// ---------------------------------------------------------------------------
// pack pass
// ---------------------------------------------------------------------------
// Item space: segment s = 2*instance + operand covers rows/128 x kt items,
// ordered row block major, K slice minor.  CTA b packs the contiguous items
// [b*per_cta, (b+1)*per_cta): one binary search for its first segment, then
// an incremental walk, and neighbouring items read neighbouring memory.
// Where item `it` of segment `sg` reads and writes.
struct PackItem {
    const Inst *I;
    int op, kb, tr;
    int64_t r0, k0, rows, rows_alloc, ld, K;
    const float *src;
    bool transposed, vec;
};

__device__ __forceinline__ PackItem pack_item(const Inst *insts, int sgi, int kb, int64_t rblock) {
    PackItem q;
    q.I = insts + (sgi >> 1);
    const Inst &I = *q.I;
    q.op = sgi & 1;
    q.kb = kb;
    q.r0 = rblock * kPackRows;
    q.k0 = (int64_t)q.kb * kPackBK;
    q.rows = q.op ? I.N : I.M;
    q.tr = q.op ? I.bn : BM;
    q.rows_alloc = q.op ? (int64_t)I.nt * I.bn : (int64_t)I.mt * BM;
    q.transposed = q.op ? (I.tb == 0) : (I.ta != 0);
    q.src = q.op ? I.src_b : I.src_a;
    q.ld = q.op ? I.ldb : I.lda;
    q.vec = (q.ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(q.src) & 15) == 0);
    q.K = I.K;
    return q;
}

// A place in the item space, advanced item by item without divisions.
struct PackCursor {
    const Inst *insts;
    const int64_t *seg_start;
    int64_t it, rblock;
    int sgi, kb, kt;

    // the item `at` of segment `sg` (at < seg_start[sg + 1])
    __device__ __forceinline__ void place(const Inst *in, const int64_t *starts, int sg, int64_t at) {
        insts = in, seg_start = starts, it = at, sgi = sg;
        kt = insts[sgi >> 1].kt;
        const int64_t local = it - seg_start[sgi];
        rblock = local / kt;
        kb = (int)(local - rblock * kt);
    }
    __device__ __forceinline__ PackItem item() const { return pack_item(insts, sgi, kb, rblock); }
    // to the next item, which is before `end`, the end of this CTA's range
    __device__ __forceinline__ void next(int64_t end) {
        if (++it >= end) return;
        if (++kb == kt) {
            kb = 0;
            ++rblock;
            if (it >= seg_start[sgi + 1]) {
                do ++sgi;
                while (it >= seg_start[sgi + 1]);
                kt = insts[sgi >> 1].kt;
                rblock = 0;
            }
        }
    }
};

// Stage layout: [128 rows][64 k] floats (rows of 256 B) for row-major
// sources, [64 k][128 rows] (k rows of 512 B) for transposed ones, where the
// 16-byte chunk of rows 4q..4q+3 in k row k sits at chunk q ^ ((k >> 3) & 7),
// so that the eight k-runs one warp reads per row land in distinct banks.
constexpr uint32_t kPackTileBytes = kPackRows * kPackBK * 4;
constexpr int kPackStages = 3;
constexpr uint32_t kPackSmemBytes = kPackStages * kPackTileBytes;
constexpr int kPackChunks = (int)(kPackTileBytes / 16) / 256;  // 16-byte chunks per thread per item

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(smem_dst)), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Thread `tid` copies its 16-byte chunks of item q into `stage` with async
// copies (no registers held while they fly); bytes past M, N or K are
// zero-filled by the copies themselves.
__device__ __forceinline__ void pack_issue(const PackItem &q, uint8_t *stage, int tid) {
    // stage[r][k]: 16 chunks per 256-byte row; transposed, stage[k][r]: 32 chunks
    // per 512-byte k row.  A thread keeps its chunk along the row and takes
    // every 16th row (8th k row).
    const int o = q.transposed ? tid >> 5 : tid >> 4, ostep = q.transposed ? 8 : 16;
    const int64_t outer = (q.transposed ? q.k0 : q.r0) + o;
    const int64_t inner = q.transposed ? q.r0 + (tid & 31) * 4 : q.k0 + (tid & 15) * 4;
    const int64_t left = (q.transposed ? q.rows : q.K) - inner, oleft = (q.transposed ? q.K : q.rows) - outer;
    const int inside = left >= 4 ? 4 : (left > 0 ? (int)left : 0);
    const float *p = q.src + outer * q.ld + inner;
    const int64_t step = (int64_t)ostep * q.ld;
#pragma unroll
    for (int j = 0; j < kPackChunks; ++j) {
        const int valid = j * ostep < oleft ? inside : 0;
        const float *src = valid ? p : q.src;
        uint8_t *dst = !q.transposed ? stage + (size_t)(j * 256 + tid) * 16
                                     : stage + (size_t)(o + 8 * j) * 512 + (((tid & 31) ^ j) << 4);
        if (q.vec) {
            cp_async16(dst, src, (uint32_t)valid * 4);
        } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) cp_async4(dst + 4 * v, v < valid ? src + v : q.src, v < valid ? 4u : 0u);
        }
        p += step;
    }
}

// One walk per CTA over its items: every thread keeps kPackStages - 1 items
// of async copies in flight while the CTA splits the current item from
// shared memory into BF16 pieces and writes them with 16-byte swizzled
// stores.
template <int NP>
__global__ void __launch_bounds__(256, 2) grouped_pack_kernel(const Inst *insts, const int64_t *seg_start, int nseg,
                                                           int64_t per_cta) {
    extern __shared__ __align__(128) uint8_t pack_smem[];
    const int tid = threadIdx.x;
    const int64_t nitems = seg_start[nseg];
    const int64_t it0 = (int64_t)blockIdx.x * per_cta;
    const int64_t it1 = it0 + per_cta < nitems ? it0 + per_cta : nitems;
    if (it0 >= it1) return;
    int sgi = 0;
    {
        int lo = 0, hi = nseg - 1;  // last segment whose start is <= it0
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (seg_start[mid] <= it0) lo = mid;
            else hi = mid - 1;
        }
        sgi = lo;
    }
    while (it0 >= seg_start[sgi + 1]) ++sgi;
    auto stage_of = [&](int64_t it) { return pack_smem + (size_t)((it - it0) % kPackStages) * kPackTileBytes; };

    // issue cursor: one commit group per item (empty past the range), so that
    // wait_group counts items
    PackCursor ahead, here;
    ahead.place(insts, seg_start, sgi, it0);
    here = ahead;
    auto issue_next = [&]() {
        if (ahead.it < it1) {
            pack_issue(ahead.item(), stage_of(ahead.it), tid);
            ahead.next(it1);
        }
        cp_async_commit();
    };
    for (int i = 0; i < kPackStages - 1; ++i) issue_next();

    for (int64_t it = it0; it < it1; ++it) {
        issue_next();  // into the stage the previous iteration released
        cp_async_wait<kPackStages - 1>();  // this thread's copies of item `it` have landed
        __syncthreads();                   // and every other thread's
        const PackItem cur = here.item();
        here.next(it1);
        const float *tile = reinterpret_cast<const float *>(stage_of(it));
        uint8_t *const *dst = cur.op ? cur.I->pb : cur.I->pa;
#pragma unroll
        for (int pass = 0; pass < kPackRows * (kPackBK / 8) / 256; ++pass) {
            const int e = pass * 256 + tid;
            // 8 threads per row (coalesced 128-byte runs of pieces), 4 rows per warp
            const int r = e >> 3, c = e & 7;
            const int64_t row = cur.r0 + r;
            if (row >= cur.rows_alloc) continue;
            float x[8];
            if (!cur.transposed) {
                // the upper four threads read their second half first: no bank conflicts
                const int h = (c >> 2) & 1;
                const float4 u = *reinterpret_cast<const float4 *>(tile + r * kPackBK + c * 8 + 4 * h);
                const float4 v = *reinterpret_cast<const float4 *>(tile + r * kPackBK + c * 8 + 4 * (h ^ 1));
                const float4 lo = h ? v : u, hi = h ? u : v;
                x[0] = lo.x, x[1] = lo.y, x[2] = lo.z, x[3] = lo.w, x[4] = hi.x, x[5] = hi.y, x[6] = hi.z, x[7] = hi.w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int k = c * 8 + j;  // (k >> 3) & 7 == c
                    x[j] = tile[k * kPackRows + ((((r >> 2) ^ c) << 2) | (r & 3))];
                }
            }
            __nv_bfloat16 pcs[8][3];
#pragma unroll
            for (int j = 0; j < 8; ++j) tcg::split_value<NP>(x[j], pcs[j]);
            const int64_t off = packed_offset(row, cur.kb, c, cur.tr, cur.I->kt);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __nv_bfloat162 v = __halves2bfloat162(pcs[2 * j][i], pcs[2 * j + 1][i]);
                    w[j] = *reinterpret_cast<uint32_t *>(&v);
                }
                *reinterpret_cast<uint4 *>(dst[i] + off) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        __syncthreads();  // this stage is read: the next issue may refill it
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// persistent contraction
// ---------------------------------------------------------------------------
struct Params {
    const TileRec *tiles;
    const int32_t *cta_start;  // tiles of CTA (pair kernel: cluster) b: [cta_start[b], cta_start[b+1])
    int seg_kblocks;
    int *fault;
};

// PAIR: a cluster of two CTAs runs 256 x bn tiles (an instance's row blocks
// in pairs), the leader issuing cta_group::2 MMAs (M = 256) on both CTAs'
// shared memory: each CTA stages its own 128-row A tile and half of the B
// tile's rows, so at bn = 256 a CTA moves a third fewer operand bytes per MMA
// than on a single-CTA 128 x 256 tile.
// Each CTA's copies complete on its own barrier; the peer's warp 1 relays
// every landed stage to the leader's barrier, which the MMA issuer waits on.
// The leader's MMAs commit to both CTAs' ring and accumulator barriers; both
// CTAs' drain warps (each on its own 128 rows of TMEM) arrive on the leader's.
//
// The epilogue bounds short-K tiles: C is read and written once per tile, and
// what counts is how much of it a warp has in flight and how whole its lines
// are.  Sums are kept a row per lane (32x32b reads) and go through a 4 KiB
// staging tile per warp, so that each instruction moves VEC rows of a 32-column
// chunk by VEC floats a lane, with all the chunk's reads of C (4 KiB a warp) in
// flight together.  VEC is 4, 2 or 1: all instances' N, ldc and C are multiples
// of it.  Before, reads and stores were 32-byte pieces of eight rows, two
// floats a lane, or one at a time when N was odd.  Contraction only, BF16, 148
// products of 1024 x N x 128, beta = 1, N = 1024 / 1022 / 1023: 273 -> 227, 320
// -> 274, 1590 -> 325 us; with beta = 0 162 -> 147, 217 -> 222 (lines split
// between rows bound it), 370 -> 235 us.  256 uneven products up to 2048: split3 180
// -> 166, BF16 118 -> 103 us.
template <int VEC> struct alignas(4 * VEC) Vec { float x[VEC]; };

template <int MODE, bool PAIR, int VEC>
__global__ void __launch_bounds__(kThreads, 1) grouped_gemm_kernel(Params p) {
    using L = GLayoutOf<MODE, PAIR>;
    using MD = tcg::Mode<MODE>;
    constexpr int S = L::STAGES;
    static_assert(L::BK == kBK, "grouped engine stages BF16 slices of kBK");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[S], empty[S], tfull[2], tempty[2], mma_done;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ int ring_issued, ring_consumed, mma_aborted;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? tc::cluster_ctarank() : 0u;
    const bool leader = rank == 0;
    const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int t_begin = p.cta_start[unit], t_end = p.cta_start[unit + 1];
    auto wait_lane = [&](uint64_t *bar, uint32_t parity, uint64_t limit) {
        return PAIR ? tc::wait_timed_cluster(bar, parity, limit, &abort_flag)
                    : tc::wait_timed(bar, parity, limit, &abort_flag);
    };
    auto wait_warp = [&](uint64_t *bar, uint32_t parity, uint64_t limit) {
        return PAIR ? tc::wait_warp_cluster(bar, parity, limit, &abort_flag)
                    : tc::wait_warp(bar, parity, limit, &abort_flag);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            // the leader's stage completes on its own copies and the peer's relay
            mbar_init(&full[s], PAIR && leader ? 2 : 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], (PAIR ? 2 : 1) * kDrainWarps);
        }
        mbar_init(&mma_done, 1);
        fence_mbarrier_init();
        abort_flag = 0;
        ring_issued = ring_consumed = 0;
        mma_aborted = 0;
    }
    if (warp == 0) {
        if constexpr (PAIR) {
            tc::tmem_alloc_pair(&tmem_base, kTmemCols);
            tc::tmem_relinquish_pair();
        } else {
            tc::tmem_alloc(&tmem_base, kTmemCols);
            tc::tmem_relinquish();
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if constexpr (PAIR) tc::cluster_sync();  // both CTAs' barriers exist before any signal crosses the pair
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;

    auto a_tile = [&](int s, int piece) { return smem + s * L::STAGE_BYTES + piece * L::A_TILE; };
    auto b_tile = [&](int s, int piece) { return smem + s * L::STAGE_BYTES + MD::NP * L::A_TILE + piece * L::B_TILE; };

    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    if (warp == 0) {
        // ---- producer: one bulk copy per piece tile (all lanes walk and wait,
        // one elected lane issues, as in the MMA warp) ----
        int ring = 0, s = 0;
        uint32_t ph = 0;
        bool stop = false;
        TileRec cur;
        if (t_begin < t_end) cur = p.tiles[t_begin];
        for (int t = t_begin; t < t_end && !stop; ++t) {
            // the next record loads while this tile's copies are issued
            const TileRec next = p.tiles[t + 1 < t_end ? t + 1 : t];
            // a slice of the B tile is bn rows, and a pair CTA copies its half of
            // them; rank 1's A tile is the next row block, or (in a tile of 128
            // rows or fewer) rank 0's again, whose products are never stored
            const uint32_t b_slice = (uint32_t)cur.bn * kRowBytes;
            const uint32_t b_bytes = PAIR ? b_slice / 2 : b_slice;
            const int64_t a_off = (PAIR && rank == 1 && cur.rows > BM) ? (int64_t)cur.kt * kATileBytes : 0;
            const int64_t b_off = PAIR ? (int64_t)rank * b_bytes : 0;
            for (int kb = 0; kb < cur.kt; ++kb, ++ring) {
                if (!wait_warp(&empty[s], ph ^ 1u, kWaitNs)) {
                    if (lane == 0) {
                        if (!abort_flag) report_fault(p.fault, kFaultTcProducerWait);
                        abort_flag = 1;
                    }
                    stop = true;
                    break;
                }
                if (tc::elect_one()) {
                    mbar_arrive_expect_tx(&full[s], MD::NP * (kATileBytes + b_bytes));
                    for (int i = 0; i < MD::NP; ++i) {
                        bulk_g2s(a_tile(s, i), cur.a[i] + a_off + (int64_t)kb * kATileBytes, kATileBytes, &full[s]);
                        bulk_g2s(b_tile(s, i), cur.b[i] + b_off + (int64_t)kb * b_slice, b_bytes, &full[s]);
                    }
                }
                __syncwarp();
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            cur = next;
        }
        if (lane == 0) ring_issued = ring;
        __syncwarp();
    } else if (warp == 1) {
        if (PAIR && !leader && lane == 0) {
            // ---- relay: each landed stage of this CTA, to the leader's barrier ----
            const uint32_t full_leader = tc::mapa_shared(smem_u32(&full[0]), 0);
            int ring = 0;
            bool stop = false;
            for (int t = t_begin; t < t_end && !stop; ++t) {
                const int kt = p.tiles[t].kt;
                for (int kb = 0; kb < kt; ++kb, ++ring) {
                    const int s = ring % S;
                    if (!wait_lane(&full[s], (uint32_t)(ring / S) & 1u, kWaitNs)) {
                        if (!abort_flag) report_fault(p.fault, kFaultTcProducerWait);
                        abort_flag = 1;
                        stop = true;
                        break;
                    }
                    tc::mbar_arrive_remote(full_leader + (uint32_t)(s * sizeof(uint64_t)));
                }
            }
        } else if (!PAIR || leader) {
            // ---- MMA issuer: the whole warp walks the slices, so that addresses
            // and descriptors stay in uniform registers, and one elected lane
            // issues: under `lane == 0` each MMA's operands are moved there
            // first, which takes longer than an MMA of width 64 or 128 ----
            const uint64_t desc0 = tc::smem_desc_kmajor(smem_u32(smem), L::SBO, L::SWIZZLE);
            const uint32_t empty_self = PAIR ? tc::mapa_shared(smem_u32(&empty[0]), 0) : 0u;
            const uint32_t empty_peer = PAIR ? tc::mapa_shared(smem_u32(&empty[0]), 1) : 0u;
            const uint32_t tfull_self = PAIR ? tc::mapa_shared(smem_u32(&tfull[0]), 0) : 0u;
            const uint32_t tfull_peer = PAIR ? tc::mapa_shared(smem_u32(&tfull[0]), 1) : 0u;
            int ring = 0, seg = 0, s = 0;
            uint32_t ph = 0;
            bool stop = false;
            int2 cur = make_int2(0, 0);  // (kt, bn)
            if (t_begin < t_end) cur = make_int2(p.tiles[t_begin].kt, p.tiles[t_begin].bn);
            for (int t = t_begin; t < t_end && !stop; ++t) {
                const int tn = t + 1 < t_end ? t + 1 : t;
                const int2 next = make_int2(p.tiles[tn].kt, p.tiles[tn].bn);
                const int kt = __shfl_sync(0xffffffffu, cur.x, 0);
                const uint32_t idesc = tc::idesc_bf16_f32(PAIR ? 2 * BM : BM, __shfl_sync(0xffffffffu, cur.y, 0));
                cur = next;
                int in_seg = 0;  // slices of the current segment issued
                for (int kb = 0; kb < kt; ++kb, ++ring) {
                    const int b = seg & 1;
                    const bool seg_first = in_seg == 0;
                    const bool seg_last = ++in_seg == p.seg_kblocks || kb == kt - 1;
                    if ((seg_first && !wait_warp(&tempty[b], ((uint32_t)(seg >> 1) & 1u) ^ 1u, kWaitNs)) ||
                        !wait_warp(&full[s], ph, kWaitNs)) {
                        if (lane == 0) {
                            if (!abort_flag) report_fault(p.fault, kFaultTcMmaWait);
                            abort_flag = 1;
                        }
                        stop = true;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t d = tmem + (uint32_t)(b * 256);
                    const uint64_t at = desc0 + (uint64_t)(s * (L::STAGE_BYTES >> 4));
                    const uint64_t bt = at + ((MD::NP * L::A_TILE) >> 4);
                    if (tc::elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < L::KSTEPS; ++kk) {
#pragma unroll
                            for (int j = 0; j < MD::NPROD; ++j) {
                                const uint64_t ad = at + ((MD::pa(j) * L::A_TILE + kk * 32) >> 4);
                                const uint64_t bd = bt + ((MD::pb(j) * L::B_TILE + kk * 32) >> 4);
                                const uint32_t accum = (seg_first && kk == 0 && j == 0) ? 0u : 1u;
                                if constexpr (PAIR) tc::mma_bf16_pair(d, ad, bd, idesc, accum);
                                else tc::mma_bf16(d, ad, bd, idesc, accum);
                            }
                        }
                        if constexpr (PAIR) {
                            const uint32_t so = (uint32_t)(s * sizeof(uint64_t)), bo = (uint32_t)(b * sizeof(uint64_t));
                            tc::commit_pair_to(empty_self + so);
                            tc::commit_pair_to(empty_peer + so);
                            if (seg_last) {
                                tc::commit_pair_to(tfull_self + bo);
                                tc::commit_pair_to(tfull_peer + bo);
                            }
                        } else {
                            tc::commit_to(&empty[s]);
                            if (seg_last) tc::commit_to(&tfull[b]);
                        }
                    }
                    __syncwarp();
                    if (seg_last) {
                        ++seg;
                        in_seg = 0;
                    }
                    if (++s == S) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (lane == 0) ring_consumed = ring;
            if (stop && tc::elect_one()) {
                // every MMA issued before the abort completes before TMEM is freed
                mma_aborted = 1;
                if constexpr (PAIR) tc::commit_pair_to(tc::mapa_shared(smem_u32(&mma_done), 0));
                else tc::commit_to(&mma_done);
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ---- drain + epilogue ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDrainRegs));
        const int quarter = warp & 3, part = (warp - 4) >> 2;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const int row_off = PAIR ? (int)rank * 128 : 0;  // a pair CTA's rows of the 256-row tile
        const uint32_t tempty_leader = PAIR ? tc::mapa_shared(smem_u32(&tempty[0]), 0) : 0u;
        uint8_t *stage = smem + L::EPI_OFFSET + (warp - 4) * kEpiTileBytes;
        const int vr = lane / (32 / VEC), vc = lane % (32 / VEC) * VEC;  // a lane's row and column of an access to C
        int seg = 0;
        bool ok = true;
        for (int t = t_begin; t < t_end && ok; ++t) {
            const TileRec rec = p.tiles[t];
            const int bn = rec.bn, kt = rec.kt;
            const int hw = bn / kDrainParts;   // columns of this warp's part of the tile: 32, 64 or 128
            const int nseg = (kt + p.seg_kblocks - 1) / p.seg_kblocks;
            // acc[c]: row `lane` of this warp's 32, column c of its part
            float acc[kPartCols];
#pragma unroll
            for (int j = 0; j < kPartCols; ++j) acc[j] = 0.0f;
            const int row0 = row_off + quarter * 32;
            const int left = rec.cols - part * hw;
            const int ncols = left < hw ? left : hw;  // valid columns of this part (may be none)
            const int nrows = rec.rows - row0 < 32 ? rec.rows - row0 : 32;
            // without the gemm option 1 and 0: a sum that began at +0 is never -0, so 1 * sum + 0 is the sum
            const float alpha = rec.gemm ? rec.alpha : 1.0f;
            const float beta = rec.gemm && rec.beta != 0.0f ? rec.beta : 0.0f;
            float *C = rec.C + (int64_t)row0 * rec.ldc + part * hw;
            if (beta != 0.0f && lane < nrows) {
                // C is read by the epilogue: pull this warp's rows of it into L2
                // while the tile's MMAs run
                const char *row = reinterpret_cast<const char *>(C + (int64_t)lane * rec.ldc);
                for (int off = 0; off < ncols * 4; off += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + off));
            }
            for (int sg = 0; sg < nseg; ++sg, ++seg) {
                const int b = seg & 1;
                if (!wait_warp(&tfull[b], (uint32_t)(seg >> 1) & 1u, 2 * kWaitNs)) {
                    if (!abort_flag) report_fault(p.fault, kFaultTcEpilogueWait);
                    abort_flag = 1;
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t col_base = tmem + lane_base + (uint32_t)(b * 256 + part * hw);
#pragma unroll
                for (int c = 0; c < kPartCols; c += 16) {
                    if (c < hw) {
                        uint32_t r[16];
                        tc::tmem_ld_32x32b_x16(col_base + (uint32_t)c, r);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c + j] = __fadd_rn(acc[c + j], __uint_as_float(r[j]));
                    }
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    if (!PAIR || leader) mbar_arrive(&tempty[b]);
                    else tc::mbar_arrive_remote(tempty_leader + (uint32_t)(b * sizeof(uint64_t)));
                }
            }
            if (__any_sync(0xffffffffu, !ok || abort_flag)) break;
            // C by 32 x 32 chunks through the warp's staging tile (16-byte chunk j
            // of row r at j ^ (r & 7)): read and written in whole 128-byte lines
#pragma unroll
            for (int c = 0; c < kPartCols; c += 32) {
                if (c >= ncols || nrows <= 0) break;
                float *at = C + (int64_t)vr * rec.ldc + c + vc;
                const bool in = c + vc < ncols;  // N is a multiple of VEC: vectors are in or out
                Vec<VEC> old[32 / VEC];
#pragma unroll
                for (int i = 0; i < 32 / VEC; ++i) old[i] = {};
                if (beta != 0.0f) {
#pragma unroll
                    for (int i = 0; i < 32; i += VEC)
                        if (in && i + vr < nrows)
                            old[i / VEC] = *reinterpret_cast<const Vec<VEC> *>(at + i * rec.ldc);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<float4 *>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                        make_float4(acc[c + 4 * j], acc[c + 4 * j + 1], acc[c + 4 * j + 2], acc[c + 4 * j + 3]);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 32; i += VEC) {
                    const int r = i + vr;
                    Vec<VEC> v = *reinterpret_cast<const Vec<VEC> *>(
                        stage + r * 128 + (((vc >> 2) ^ (r & 7)) << 4) + (vc & 3) * 4);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) v.x[e] = __fmaf_rn(alpha, v.x[e], beta * old[i / VEC].x[e]);
                    if (in && r < nrows) *reinterpret_cast<Vec<VEC> *>(at + i * rec.ldc) = v;
                }
                __syncwarp();  // the staging tile is read
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && abort_flag) {
        if constexpr (PAIR) {
            // a pair's stages complete on two CTAs' barriers: give every copy in
            // flight time to land (microseconds), then the MMAs issued before the abort
            const uint64_t t0 = tc::globaltimer();
            while (tc::globaltimer() - t0 < 20000000ull) {
            }
            if (leader && mma_aborted) tc::wait_timed(&mma_done, 0, kWaitNs, nullptr);
        } else {
            // bounded waits for the copies still landing and the MMAs issued before the abort
            for (int r = ring_consumed; r < ring_issued; ++r)
                tc::wait_timed(&full[r % S], (uint32_t)(r / S) & 1u, kWaitNs, nullptr);
            if (mma_aborted) tc::wait_timed(&mma_done, 0, kWaitNs, nullptr);
        }
    }
    __syncthreads();
    if constexpr (PAIR) {
        tc::cluster_sync();  // neither CTA leaves while the pair can still touch its memory
        if (warp == 0) tc::tmem_dealloc_pair(tmem, kTmemCols);
    } else {
        if (warp == 0) tc::tmem_dealloc(tmem, kTmemCols);
    }
}

}  // namespace grp

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

std::mutex g_table_mu;
// per-bucket tile width, indexed [engine is split3][bucket]
int32_t g_tile_table[2][kGroupedBuckets] = {{64, 128, 256, 256}, {64, 128, 256, 256}};

int engine_slot(int engine) { return engine == GATLAS_ENGINE_TC_SPLIT3 ? 1 : 0; }

std::atomic<int> g_pair_mode{0};

size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

int32_t grouped_bucket(int64_t m, int64_t n, int64_t k) {
    (void)m;
    (void)k;
    if (n <= 64) return 0;
    if (n <= 128) return 1;
    if (n <= 256) return 2;
    return 3;
}

int grouped_set_pair(int mode) {
    if (mode < 0 || mode > 1) return set_error(GATLAS_ERR_INVALID, "grouped_pair: %d (0 single CTAs, 1 CTA pairs)", mode);
    g_pair_mode.store(mode);
    return GATLAS_OK;
}

int grouped_get_pair() { return g_pair_mode.load(); }

// Clusters of two that fit at once (occupancy query, once per device).
template <int MODE>
static int pair_units_cap() {
    static thread_local int cap_dev = -1, cap = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (cap_dev != dev) {
        auto kern = grp::grouped_gemm_kernel<MODE, true, 1>;
        cap = sm_count() / 2;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)grp::GLayoutOf<MODE, true>::SMEM_BYTES) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(2 * (unsigned)cap, 1, 1);
            cfg.blockDim = dim3(grp::kThreads, 1, 1);
            cfg.dynamicSmemBytes = grp::GLayoutOf<MODE, true>::SMEM_BYTES;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) cap = n;
        }
        cudaGetLastError();
        cap_dev = dev;
    }
    return std::max(cap, 1);
}

int grouped_set_tile_table(int engine, const int32_t *t, int32_t nb) {
    if (engine != GATLAS_ENGINE_TC_BF16 && engine != GATLAS_ENGINE_TC_SPLIT3)
        return set_error(GATLAS_ERR_UNSUPPORTED, "grouped: engine %d has no grouped kernel", engine);
    if (!t || nb != kGroupedBuckets) return set_error(GATLAS_ERR_INVALID, "grouped: tile table needs %d entries", kGroupedBuckets);
    for (int i = 0; i < nb; ++i)
        if (t[i] != 64 && t[i] != 128 && t[i] != 256) return set_error(GATLAS_ERR_INVALID, "grouped: tile width %d", t[i]);
    std::lock_guard<std::mutex> lk(g_table_mu);
    for (int i = 0; i < nb; ++i) g_tile_table[engine_slot(engine)][i] = t[i];
    return GATLAS_OK;
}

int grouped_get_tile_table(int engine, int32_t *t, int32_t nb) {
    if (engine != GATLAS_ENGINE_TC_BF16 && engine != GATLAS_ENGINE_TC_SPLIT3)
        return set_error(GATLAS_ERR_UNSUPPORTED, "grouped: engine %d has no grouped kernel", engine);
    if (!t || nb != kGroupedBuckets) return set_error(GATLAS_ERR_INVALID, "grouped: tile table needs %d entries", kGroupedBuckets);
    std::lock_guard<std::mutex> lk(g_table_mu);
    for (int i = 0; i < nb; ++i) t[i] = g_tile_table[engine_slot(engine)][i];
    return GATLAS_OK;
}

static int resolve_instance(const gatlas_grouped_instance &in, int slot, InstPlan *o) {
    if (in.m < 0 || in.n < 0 || in.k < 0) return set_error(GATLAS_ERR_INVALID, "grouped: negative dimension");
    o->M = in.m, o->N = in.n, o->K = in.k;
    const int64_t a_inner = in.trans_a ? in.m : in.k, b_inner = in.trans_b ? in.k : in.n;
    o->lda = in.lda ? in.lda : std::max<int64_t>(a_inner, 1);
    o->ldb = in.ldb ? in.ldb : std::max<int64_t>(b_inner, 1);
    o->ldc = in.ldc ? in.ldc : std::max<int64_t>(in.n, 1);
    if (o->lda < a_inner || o->ldb < b_inner || o->ldc < in.n)
        return set_error(GATLAS_ERR_INVALID, "grouped: leading dimension below the stored row length");
    int bn = in.tile_n;
    if (bn == 0) {
        std::lock_guard<std::mutex> lk(g_table_mu);
        bn = g_tile_table[slot][grouped_bucket(in.m, in.n, in.k)];
    }
    if (bn != 64 && bn != 128 && bn != 256) return set_error(GATLAS_ERR_INVALID, "grouped: tile width %d", bn);
    o->bn = bn;
    o->mt = (int)((in.m + grp::BM - 1) / grp::BM);
    o->nt = (int)((in.n + bn - 1) / bn);
    o->kt = (int)((in.k + grp::kPackBK - 1) / grp::kPackBK);
    if (in.m == 0 || in.n == 0) o->mt = o->nt = 0;
    if (o->mt > 65535 || o->kt > (1 << 24)) return set_error(GATLAS_ERR_INVALID, "grouped: instance too large");
    o->a_piece = round_up((size_t)o->mt * o->kt * grp::BM * grp::kPackRowBytes, 1024);
    o->b_piece = round_up((size_t)o->nt * o->kt * bn * grp::kPackRowBytes, 1024);
    return GATLAS_OK;
}

static bool grouped_engine_ok(int engine) {
    return engine == GATLAS_ENGINE_TC_BF16 || engine == GATLAS_ENGINE_TC_SPLIT3;
}

int grouped_instance_bytes(int engine, const gatlas_grouped_instance &in, size_t *bytes) {
    if (!grouped_engine_ok(engine))
        return set_error(GATLAS_ERR_UNSUPPORTED, "grouped: engine %d has no grouped kernel (tc_bf16, tc_split3)", engine);
    InstPlan o{};
    const int rc = resolve_instance(in, engine_slot(engine), &o);
    if (rc) return rc;
    const int np = engine == GATLAS_ENGINE_TC_SPLIT3 ? 2 : 1;
    *bytes = np * (o.a_piece + o.b_piece);
    return GATLAS_OK;
}

int grouped_build(int engine, const gatlas_grouped_instance *in, int32_t count, uint8_t *base,
                  uint8_t *const *packed, GroupedTables *t) {
    if (!grouped_engine_ok(engine))
        return set_error(GATLAS_ERR_UNSUPPORTED, "grouped: engine %d has no grouped kernel (tc_bf16, tc_split3)", engine);
    if (count < 0 || (count > 0 && !in)) return set_error(GATLAS_ERR_INVALID, "grouped: invalid instance list");
    t->engine = engine;
    t->np = engine == GATLAS_ENGINE_TC_SPLIT3 ? 2 : 1;
    t->mode = engine == GATLAS_ENGINE_TC_SPLIT3 ? 1 : 0;
    t->ip.assign(count, InstPlan{});
    t->inst.assign(std::max(count, 1), grp::Inst{});
    t->seg.assign(2 * (size_t)count + 1, 0);
    t->flops = 0;
    t->packed_bytes = 0;
    struct Cand {
        int64_t cost;
        grp::TileRec r;
    };
    std::vector<Cand> cands;
    for (int i = 0; i < count; ++i) {
        int rc = resolve_instance(in[i], engine_slot(engine), &t->ip[i]);
        if (rc) return rc;
    }
    t->pair = g_pair_mode.load() == 1;
    // the widest access to C that every instance takes
    uint64_t low = 0;  // bits set in any N, ldc or C (in floats)
    int64_t c_elems = 0;
    bool reads_c = false;
    for (int i = 0; i < count; ++i)
        if (in[i].m > 0 && in[i].n > 0) {
            low |= (uint64_t)t->ip[i].N | (uint64_t)t->ip[i].ldc | reinterpret_cast<uintptr_t>(in[i].c) >> 2;
            c_elems += (int64_t)in[i].m * in[i].n;
            reads_c = reads_c || (in[i].gemm && in[i].beta != 0.0);
        }
    t->vec = low & 1 ? 1 : low & 2 ? 2 : 4;
    // Written only, and more than L2 holds: one float a lane, a whole row of a chunk
    // per access.  Two rows per access leave more sectors of rows off the 16-byte
    // grid for later (148 products of 1024 x 1022 x 128 BF16 208 us, 243 with pairs;
    // 256 of 256 x 254 x 256, in L2, 39 and 34).
    if (t->vec == 2 && !reads_c && c_elems > (32ll << 20)) t->vec = 1;
    const int step_m = t->pair ? 2 : 1;
    size_t off = 0;
    for (int i = 0; i < count; ++i) {
        InstPlan &o = t->ip[i];
        const gatlas_grouped_instance &q = in[i];
        if (q.m > 0 && q.n > 0 && (!q.c || (q.k > 0 && (!q.a || !q.b))))
            return set_error(GATLAS_ERR_INVALID, "grouped: instance %d has a null pointer", i);
        uint8_t *pb = packed ? packed[i] : (base ? base + off : nullptr);
        off += t->np * (o.a_piece + o.b_piece);
        t->packed_bytes += t->np * (o.a_piece + o.b_piece);
        t->flops += 2.0 * (double)q.m * (double)q.n * (double)q.k;
        grp::Inst &I = t->inst[i];
        std::memset(&I, 0, sizeof(I));
        I.src_a = q.a;
        I.src_b = q.b;
        for (int j = 0; j < t->np && pb; ++j) {
            I.pa[j] = pb + j * o.a_piece;
            I.pb[j] = pb + t->np * o.a_piece + j * o.b_piece;
        }
        I.C = q.c;
        I.M = o.M, I.N = o.N, I.K = o.K, I.lda = o.lda, I.ldb = o.ldb, I.ldc = o.ldc;
        I.ta = q.trans_a != 0, I.tb = q.trans_b != 0, I.gemm = q.gemm != 0;
        I.bn = o.bn, I.mt = o.mt, I.nt = o.nt, I.kt = o.kt;
        I.alpha = (float)q.alpha;
        I.beta = (float)q.beta;
        const int64_t a_items = o.kt ? (int64_t)o.mt * o.kt : 0;  // 128 A rows per item = one A tile row block
        const int64_t b_items = o.kt ? ((int64_t)o.nt * o.bn + grp::kPackRows - 1) / grp::kPackRows * o.kt : 0;
        t->seg[2 * i + 1] = t->seg[2 * i] + a_items;
        t->seg[2 * i + 2] = t->seg[2 * i + 1] + b_items;
        // cost in bytes moved: operand tiles through shared memory plus the C
        // tile (read too when beta != 0), plus a fixed per-tile overhead
        // (a pair tile: both CTAs' halves, as one unit of its cluster's time)
        const int64_t c_bytes = (int64_t)step_m * grp::BM * o.bn * 4 * ((q.gemm && q.beta != 0.0) ? 2 : 1);
        const int64_t cost = (int64_t)o.kt * t->np * (step_m * grp::BM + o.bn) * grp::kPackRowBytes + c_bytes + 16384;
        // grouped raster inside the instance: 16 tile rows per group, so the
        // tiles that run at the same time share A and B rows through L2
        for (int g0 = 0; g0 < o.mt; g0 += 16)
            for (int tn = 0; tn < o.nt; ++tn)
                for (int tm = g0; tm < std::min(o.mt, g0 + 16); tm += step_m) {
                grp::TileRec r;
                std::memset(&r, 0, sizeof(r));
                for (int j = 0; j < t->np && pb; ++j) {
                    r.a[j] = I.pa[j] + (size_t)tm * o.kt * grp::BM * grp::kPackRowBytes;
                    r.b[j] = I.pb[j] + (size_t)tn * o.kt * o.bn * grp::kPackRowBytes;
                }
                r.C = q.c + (int64_t)tm * grp::BM * o.ldc + (int64_t)tn * o.bn;
                r.ldc = o.ldc;
                r.kt = o.kt * grp::kSlicesPerItem;  // contraction K slices
                r.bn = o.bn;
                r.rows = (int32_t)std::min<int64_t>(step_m * grp::BM, o.M - (int64_t)tm * grp::BM);
                r.cols = (int32_t)std::min<int64_t>(o.bn, o.N - (int64_t)tn * o.bn);
                r.alpha = (float)q.alpha;
                r.beta = (float)q.beta;
                r.gemm = q.gemm != 0;
                cands.push_back(Cand{cost, r});
            }
    }
    t->nseg = 2 * count;
    t->nitems = t->seg.back();
    t->ntiles = (int64_t)cands.size();
    // longest first onto the least-loaded CTA
    std::stable_sort(cands.begin(), cands.end(), [](const Cand &a, const Cand &b) { return a.cost > b.cost; });
    const int units = t->pair ? (t->mode == 1 ? pair_units_cap<1>() : pair_units_cap<0>()) : sm_count();
    t->grid = (int)std::min<int64_t>(units, std::max<int64_t>(t->ntiles, 1));
    std::vector<int> owner(cands.size());
    std::vector<int32_t> count_per(t->grid, 0);
    {
        using E = std::pair<int64_t, int>;
        std::priority_queue<E, std::vector<E>, std::greater<E>> heap;
        for (int b = 0; b < t->grid; ++b) heap.push({0, b});
        for (size_t c = 0; c < cands.size(); ++c) {
            E e = heap.top();
            heap.pop();
            owner[c] = e.second;
            ++count_per[e.second];
            heap.push({e.first + cands[c].cost, e.second});
        }
    }
    t->cta.assign(t->grid + 1, 0);
    for (int b = 0; b < t->grid; ++b) t->cta[b + 1] = t->cta[b] + count_per[b];
    t->tiles.assign(std::max<size_t>(cands.size(), 1), grp::TileRec{});
    std::vector<int32_t> fill(t->cta.begin(), t->cta.end() - 1);
    for (size_t c = 0; c < cands.size(); ++c) t->tiles[fill[owner[c]]++] = cands[c].r;
    return GATLAS_OK;
}

// Shared-memory attribute of the pack kernels, once per device (also before
// a graph capture, since attribute changes are not captured).
static void grouped_pack_attributes() {
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev == dev) return;
    cudaFuncSetAttribute(grp::grouped_pack_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)grp::kPackSmemBytes);
    cudaFuncSetAttribute(grp::grouped_pack_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)grp::kPackSmemBytes);
    attr_dev = dev;
}

int grouped_launch_pack(const GroupedTables &t, const GroupedDevice &d, cudaStream_t stream) {
    if (t.nitems == 0) return GATLAS_OK;
    // two resident CTAs per SM (96 KiB of staging each), one item range per CTA
    grouped_pack_attributes();
    const int64_t grid = std::min<int64_t>(t.nitems, (int64_t)sm_count() * 2);
    const int64_t per_cta = (t.nitems + grid - 1) / grid;
    if (t.np == 2)
        grp::grouped_pack_kernel<2><<<(unsigned)grid, 256, grp::kPackSmemBytes, stream>>>(d.inst, d.seg, t.nseg,
                                                                                          per_cta);
    else
        grp::grouped_pack_kernel<1><<<(unsigned)grid, 256, grp::kPackSmemBytes, stream>>>(d.inst, d.seg, t.nseg,
                                                                                          per_cta);
    return check_launch("grouped_pack_kernel");
}

// Shared-memory attributes of the contraction kernels, once per device (also
// before a graph capture, since attribute changes are not captured).
template <int MODE, bool PAIR>
static cudaError_t grouped_gemm_attribute() {
    const int bytes = (int)grp::GLayoutOf<MODE, PAIR>::SMEM_BYTES;
    for (auto kern : {grp::grouped_gemm_kernel<MODE, PAIR, 1>, grp::grouped_gemm_kernel<MODE, PAIR, 2>,
                      grp::grouped_gemm_kernel<MODE, PAIR, 4>}) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

static int grouped_gemm_attributes() {
    static thread_local int attr_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev == dev) return GATLAS_OK;
    for (cudaError_t e : {grouped_gemm_attribute<0, false>(), grouped_gemm_attribute<1, false>(),
                          grouped_gemm_attribute<0, true>(), grouped_gemm_attribute<1, true>()})
        if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "grouped smem attribute: %s", cudaGetErrorString(e));
    attr_dev = dev;
    return GATLAS_OK;
}

template <int MODE, bool PAIR>
static int launch_grouped(const GroupedTables &t, const GroupedDevice &d, cudaStream_t stream) {
    grp::Params prm;
    prm.tiles = d.tiles;
    prm.cta_start = d.cta;
    prm.seg_kblocks = grp::grouped_seg_kblocks(MODE);
    prm.fault = device_fault_word();
    const int rc = grouped_gemm_attributes();
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((PAIR ? 2 : 1) * t.grid), 1, 1);
    cfg.blockDim = dim3(grp::kThreads, 1, 1);
    cfg.dynamicSmemBytes = grp::GLayoutOf<MODE, PAIR>::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = PAIR ? 1 : 0;
    const auto kern = t.vec == 4   ? grp::grouped_gemm_kernel<MODE, PAIR, 4>
                      : t.vec == 2 ? grp::grouped_gemm_kernel<MODE, PAIR, 2>
                                   : grp::grouped_gemm_kernel<MODE, PAIR, 1>;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, prm);
    if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "grouped_gemm_kernel: %s", cudaGetErrorString(e));
    return check_launch("grouped_gemm_kernel");
}

int grouped_launch_contract(const GroupedTables &t, const GroupedDevice &d, cudaStream_t stream) {
    if (t.ntiles == 0) return GATLAS_OK;
    if (t.pair) return t.mode == 1 ? launch_grouped<1, true>(t, d, stream) : launch_grouped<0, true>(t, d, stream);
    return t.mode == 1 ? launch_grouped<1, false>(t, d, stream) : launch_grouped<0, false>(t, d, stream);
}

struct GroupedPlan {
    int count = 0;
    std::vector<gatlas_grouped_instance> in;
    GroupedTables t;
    GroupedDevice d;
    void *dev_tables = nullptr;
    void *ws = nullptr;
    bool owns_ws = false;
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
};

size_t grouped_workspace_bytes(int engine, const gatlas_grouped_instance *in, int32_t count) {
    if (!grouped_engine_ok(engine) || !in || count < 0) return 0;
    size_t total = 0;
    for (int i = 0; i < count; ++i) {
        size_t b = 0;
        if (grouped_instance_bytes(engine, in[i], &b)) return 0;
        total += b;
    }
    return total;
}

static void free_plan(GroupedPlan *p) {
    for (auto &g : p->graph)
        if (g) cudaGraphExecDestroy(g);
    cudaFree(p->dev_tables);
    if (p->owns_ws) cudaFree(p->ws);
    delete p;
}

// Byte layout of the device tables: [inst][seg][tiles][cta], 256-byte aligned parts.
static size_t table_layout(const GroupedTables &t, size_t off[4]) {
    const size_t sz[4] = {t.inst.size() * sizeof(grp::Inst), t.seg.size() * sizeof(int64_t),
                          t.tiles.size() * sizeof(grp::TileRec), t.cta.size() * sizeof(int32_t)};
    size_t o = 0;
    for (int i = 0; i < 4; ++i) {
        off[i] = o;
        o += round_up(sz[i], 256);
    }
    return o;
}

size_t grouped_tables_bytes(const GroupedTables &t) {
    size_t off[4];
    return table_layout(t, off);
}

void grouped_tables_serialise(const GroupedTables &t, void *host_dst) {
    size_t off[4];
    table_layout(t, off);
    uint8_t *h = static_cast<uint8_t *>(host_dst);
    std::memcpy(h + off[0], t.inst.data(), t.inst.size() * sizeof(grp::Inst));
    std::memcpy(h + off[1], t.seg.data(), t.seg.size() * sizeof(int64_t));
    std::memcpy(h + off[2], t.tiles.data(), t.tiles.size() * sizeof(grp::TileRec));
    std::memcpy(h + off[3], t.cta.data(), t.cta.size() * sizeof(int32_t));
}

GroupedDevice grouped_tables_device(const GroupedTables &t, const void *dev_base) {
    size_t off[4];
    table_layout(t, off);
    const uint8_t *b = static_cast<const uint8_t *>(dev_base);
    GroupedDevice d;
    d.inst = reinterpret_cast<const grp::Inst *>(b + off[0]);
    d.seg = reinterpret_cast<const int64_t *>(b + off[1]);
    d.tiles = reinterpret_cast<const grp::TileRec *>(b + off[2]);
    d.cta = reinterpret_cast<const int32_t *>(b + off[3]);
    return d;
}

int grouped_create(int engine, const gatlas_grouped_instance *in, int32_t count, void *ws, size_t ws_bytes,
                   GroupedPlan **out) {
    if (!out) return set_error(GATLAS_ERR_INVALID, "grouped: null plan pointer");
    *out = nullptr;
    GroupedPlan *p = new GroupedPlan();
    p->count = count;
    if (count > 0 && in) p->in.assign(in, in + count);
    // validate and size before any device work
    int rc = grouped_build(engine, in, count, nullptr, nullptr, &p->t);
    if (rc) {
        delete p;
        return rc;
    }
    const size_t total = p->t.packed_bytes;
    if (ws) {
        if (ws_bytes < total) {
            delete p;
            return set_error(GATLAS_ERR_INVALID, "grouped: workspace %zu < %zu bytes", ws_bytes, total);
        }
        if (!aligned_to(ws, 1024)) {
            delete p;
            return set_error(GATLAS_ERR_INVALID, "grouped: workspace must be 1024-byte aligned");
        }
        p->ws = ws;
    } else if (total) {
        if (cudaMalloc(&p->ws, total) != cudaSuccess) {
            cudaGetLastError();
            delete p;
            return set_error(GATLAS_ERR_NOMEM, "grouped: workspace of %zu bytes", total);
        }
        p->owns_ws = true;
    }
    rc = grouped_build(engine, in, count, static_cast<uint8_t *>(p->ws), nullptr, &p->t);
    if (rc) {
        free_plan(p);
        return rc;
    }
    const size_t tb = grouped_tables_bytes(p->t);
    std::vector<uint8_t> host(tb);
    grouped_tables_serialise(p->t, host.data());
    if (cudaMalloc(&p->dev_tables, tb) != cudaSuccess ||
        cudaMemcpy(p->dev_tables, host.data(), tb, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        free_plan(p);
        return set_error(GATLAS_ERR_NOMEM, "grouped: device tables");
    }
    p->d = grouped_tables_device(p->t, p->dev_tables);
    *out = p;
    return GATLAS_OK;
}

int grouped_prepare(GroupedPlan *p, cudaStream_t stream) {
    if (!p) return set_error(GATLAS_ERR_INVALID, "grouped: null plan");
    return grouped_launch_pack(p->t, p->d, stream);
}

int grouped_run(GroupedPlan *p, cudaStream_t stream) {
    if (!p) return set_error(GATLAS_ERR_INVALID, "grouped: null plan");
    return grouped_launch_contract(p->t, p->d, stream);
}

int grouped_launch_graph(GroupedPlan *p, int with_prepare, cudaStream_t stream) {
    if (!p) return set_error(GATLAS_ERR_INVALID, "grouped: null plan");
    const int slot = with_prepare ? 1 : 0;
    if (!p->graph[slot]) {
        cudaStream_t cap;
        if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess)
            return set_error(GATLAS_ERR_CUDA, "grouped: capture stream");
        // attribute changes are not captured: set them before the capture
        const int arc = grouped_gemm_attributes();
        if (arc) {
            cudaStreamDestroy(cap);
            return arc;
        }
        grouped_pack_attributes();
        device_fault_word();
        cudaGraph_t graph = nullptr;
        int rc = GATLAS_OK;
        if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaStreamDestroy(cap);
            return set_error(GATLAS_ERR_CUDA, "grouped: begin capture");
        }
        if (with_prepare) rc = grouped_prepare(p, cap);
        if (!rc) rc = grouped_run(p, cap);
        cudaError_t e = cudaStreamEndCapture(cap, &graph);
        cudaStreamDestroy(cap);
        if (rc) {
            if (graph) cudaGraphDestroy(graph);
            return rc;
        }
        if (e != cudaSuccess || !graph) return set_error(GATLAS_ERR_CUDA, "grouped: end capture: %s", cudaGetErrorString(e));
        e = cudaGraphInstantiate(&p->graph[slot], graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            p->graph[slot] = nullptr;
            return set_error(GATLAS_ERR_CUDA, "grouped: graph instantiate: %s", cudaGetErrorString(e));
        }
    }
    if (cudaGraphLaunch(p->graph[slot], stream) != cudaSuccess) return check_launch("grouped graph launch");
    return GATLAS_OK;
}

static gatlas_matmul_desc instance_desc(const GroupedPlan *p, int i) {
    const gatlas_grouped_instance &q = p->in[i];
    gatlas_matmul_desc d;
    std::memset(&d, 0, sizeof(d));
    d.engine = p->t.engine;
    d.gemm = q.gemm;
    d.trans_a = q.trans_a;
    d.trans_b = q.trans_b;
    d.m = q.m, d.n = q.n, d.k = q.k;
    d.lda = p->t.ip[i].lda, d.ldb = p->t.ip[i].ldb, d.ldc = p->t.ip[i].ldc;
    d.batch = 1;
    d.alpha = q.alpha;
    d.beta = q.beta;
    return d;
}

// The comparator: one engine call (split A, split B, contraction) per
// instance, through the library's scratch buffer, grown once up front.
int grouped_run_each(GroupedPlan *p, cudaStream_t stream) {
    if (!p) return set_error(GATLAS_ERR_INVALID, "grouped: null plan");
    size_t need = 0;
    for (int i = 0; i < p->count; ++i) {
        const gatlas_matmul_desc d = instance_desc(p, i);
        need = std::max(need, gatlas_matmul_workspace_size(&d));
    }
    if (need && !device_scratch(need)) return set_error(GATLAS_ERR_NOMEM, "grouped: scratch of %zu bytes", need);
    for (int i = 0; i < p->count; ++i) {
        const gatlas_grouped_instance &q = p->in[i];
        if (q.m == 0 || q.n == 0) continue;
        const gatlas_matmul_desc d = instance_desc(p, i);
        const int rc = gatlas_matmul_f32(&d, q.a, q.b, q.c, nullptr, 0, stream);
        if (rc) return rc;
    }
    return GATLAS_OK;
}

int grouped_info(const GroupedPlan *p, int64_t *tiles, int32_t *ctas, double *flops, int64_t *items) {
    if (!p) return set_error(GATLAS_ERR_INVALID, "grouped: null plan");
    if (tiles) *tiles = p->t.ntiles;
    if (ctas) *ctas = p->t.grid * (p->t.pair ? 2 : 1);
    if (flops) *flops = p->t.flops;
    if (items) *items = p->t.nitems;
    return GATLAS_OK;
}

void grouped_destroy(GroupedPlan *p) {
    if (p) free_plan(p);
}

}  // namespace gatlas

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

size_t gatlas_grouped_workspace_size(int engine, const gatlas_grouped_instance *inst, int32_t count) {
    return gatlas::grouped_workspace_bytes(engine, inst, count);
}

int gatlas_grouped_create(int engine, const gatlas_grouped_instance *inst, int32_t count, void *workspace,
                          size_t workspace_bytes, gatlas_grouped_plan **plan) {
    gatlas::clear_error();
    return gatlas::grouped_create(engine, inst, count, workspace, workspace_bytes,
                                  reinterpret_cast<gatlas::GroupedPlan **>(plan));
}

int gatlas_grouped_prepare(gatlas_grouped_plan *plan, void *stream) {
    gatlas::clear_error();
    return gatlas::grouped_prepare(reinterpret_cast<gatlas::GroupedPlan *>(plan), (cudaStream_t)stream);
}

int gatlas_grouped_run(gatlas_grouped_plan *plan, void *stream) {
    gatlas::clear_error();
    return gatlas::grouped_run(reinterpret_cast<gatlas::GroupedPlan *>(plan), (cudaStream_t)stream);
}

int gatlas_grouped_launch_graph(gatlas_grouped_plan *plan, int32_t with_prepare, void *stream) {
    gatlas::clear_error();
    return gatlas::grouped_launch_graph(reinterpret_cast<gatlas::GroupedPlan *>(plan), with_prepare,
                                        (cudaStream_t)stream);
}

int gatlas_grouped_run_each(gatlas_grouped_plan *plan, void *stream) {
    gatlas::clear_error();
    return gatlas::grouped_run_each(reinterpret_cast<gatlas::GroupedPlan *>(plan), (cudaStream_t)stream);
}

int gatlas_grouped_info(const gatlas_grouped_plan *plan, int64_t *tiles, int32_t *ctas, double *flops,
                        int64_t *pack_items) {
    gatlas::clear_error();
    return gatlas::grouped_info(reinterpret_cast<const gatlas::GroupedPlan *>(plan), tiles, ctas, flops, pack_items);
}

void gatlas_grouped_destroy(gatlas_grouped_plan *plan) {
    gatlas::grouped_destroy(reinterpret_cast<gatlas::GroupedPlan *>(plan));
}

int32_t gatlas_grouped_bucket(int64_t m, int64_t n, int64_t k) { return gatlas::grouped_bucket(m, n, k); }

int gatlas_grouped_set_tile_table(int engine, const int32_t *bucket_tile_n, int32_t nbuckets) {
    gatlas::clear_error();
    return gatlas::grouped_set_tile_table(engine, bucket_tile_n, nbuckets);
}

int gatlas_grouped_get_tile_table(int engine, int32_t *bucket_tile_n, int32_t nbuckets) {
    gatlas::clear_error();
    return gatlas::grouped_get_tile_table(engine, bucket_tile_n, nbuckets);
}

}  // extern "C"
