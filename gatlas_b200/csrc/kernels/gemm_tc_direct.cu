// One-launch tensor-core contraction for products of few tiles: FP32 operands
// in, C out, with no split pass and no workspace.
//
// The two-pass path (gemm_tc.cu) writes BF16 pieces of both operands to global
// memory, reads them back through TMA and tiles C by 256 columns.  For a
// product of few tiles that is three launches, 3x the operand traffic and
// mostly idle SMs: 64 x 4096 x 8192 BF16 ran its contraction on 16 CTAs (110 us
// in all against 21 us for reading the operands once), 1000 x 777 x 1100 split3
// on 16 CTA pairs (66 us).
//
// Here a CTA computes one 128 x BN tile of C (BN = 32 or 64).  Sixteen warps
// load FP32 operand slices of 64 k straight into registers, split them into
// BF16 pieces and store those into a shared-memory ring in the
// 128-byte-swizzled K-major layout the MMA descriptors read; another warp
// issues tcgen05.mma; the sixteen also promote finished K segments from TMEM
// into FP32 registers (four accumulator buffers, so a promotion never holds up
// the MMAs) and at the end pass C through shared memory, so that rows of any
// alignment are read and written in full lines.
//
// Registers and not a second shared-memory ring hold the FP32 slices in
// flight, because shared memory is what the MMAs contend for.  A slice is the
// work of 8 warps (4 where only 64 rows of A exist), and two (four) groups of
// warps take the slices in turn, so that one group's loads fly while another
// splits.  Operand layouts cost the same number of shared-memory stores: a
// warp's unit of work is 256 elements, 8 per lane, as 4 rows x 64 k read by
// 16-byte vectors (stored along k, aligned), the same 4 rows read as pairs
// (any alignment), or 32 rows x 8 k read along the rows (stored across k).
//
// What bounds it: the SM's ingest of operand lines (about 64 bytes a cycle; a
// tile column re-reads all of A from L2) and the split instructions, at 700 to
// 1800 cycles a slice against 200 to 600 for its MMAs.  64 x 4096 x 8192 BF16
// 56 us (86 two-pass with the same MMA issue), split3 69 (197); 1000 x 777 x
// 1100 split3 22 (44).
//
// Results are bit-identical to the two-pass path: same pieces, same MMA
// sequence per segment, same segments, added in the same order.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include <cuda_bf16.h>

#include "../common.cuh"
#include "../device_state.cuh"
#include "../tcgen05.cuh"
#include "gemm_engines.hpp"
#include "tc_modes.cuh"

namespace gatlas {
namespace tcg {
namespace direct {

constexpr int kSlice = 64;                 // K elements per ring stage: 128 bytes of BF16 per row
// Four warpgroups load, split and drain; the fifth holds the MMA issuer and
// gives up the registers it does not need: 512 x 112 + 128 x 32 = 640 x 96.
constexpr int kWarps = 16;
constexpr int kThreads = 32 * (kWarps + 4);
constexpr int kLaunchRegs = 96, kWorkerRegs = 112, kIssuerRegs = 32;
static_assert(kWorkerRegs * 32 * kWarps + kIssuerRegs * (kThreads - 32 * kWarps) <= kLaunchRegs * kThreads, "register split");
constexpr int kBuffers = 4;                // TMEM accumulators
constexpr uint64_t kWaitNs = 2000000000ull;

template <int V>
struct Int {
    static constexpr int value = V;
};

// How an operand's rows lie in memory.
enum Kind { kAlongVec = 0, kAlong = 1, kAcross = 2 };

struct Source {
    const float *p;
    int64_t ld, rows, stride;  // element (r, k): p[r*ld + k] along, p[k*ld + r] across
    int kind;
};

struct Args {
    Source a, b;
    float *C;
    int64_t M, N, K, ldc, stride_c;
    int tiles_m, nslices, seg, last_ksteps;  // last_ksteps: 16-deep MMA steps of the last slice
    float alpha, beta;
    int gemm;
    int *fault;
};

template <int MODE, int AM, int BN_>
struct Cfg {
    using MD = Mode<MODE>;
    static constexpr int NP = MD::NP;
    static constexpr uint32_t ROW = 128;
    static constexpr uint32_t A_TILE = 128 * ROW, B_TILE = BN_ * ROW;
    static constexpr uint32_t STAGE = NP * (A_TILE + B_TILE);
    static constexpr int FIT = (int)((226 * 1024 - 1024) / STAGE);
    static constexpr int STAGES = FIT < 4 ? FIT : 4;
    static constexpr uint32_t SMEM = STAGES * STAGE + 1024;
    // units per slice, warps that share a slice, slices in flight
    static constexpr int UA = AM / 4, UB = BN_ / 4;
    static constexpr int WPS = AM == 64 && STAGES >= 4 ? 4 : 8, GROUPS = kWarps / WPS;
    // A group's wait for a stage tells phases apart only if the stage's last
    // but one use is known to be over, which its own previous slice shows when
    // the ring is at least as deep as there are groups.
    static_assert(STAGES >= GROUPS, "ring depth");
    static constexpr int JA = UA / WPS, JB = UB / WPS;  // units of A and of B per warp
    static_assert(UA % WPS == 0 && UB % WPS == 0, "units divide among the warps of a slice");
    static constexpr int PC = BN_ * 4 / kWarps;                   // columns of C per drain thread
    static constexpr int LD = PC < 16 ? PC : 16;                  // columns per TMEM load
    static constexpr int PITCH = BN_ + 1;                         // C staging tile, floats
    static_assert(STAGES >= 2, "ring depth");
    static_assert(128 * PITCH * 4 <= (int)(STAGES * STAGE), "C staging fits the ring");
};

// Splits two values into NP words of a BF16 pair each (the pieces of
// split_value).
template <int NP>
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t (&w)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
        if (i + 1 < NP) {  // exact residuals
            x0 -= __uint_as_float(w[i] << 16);
            x1 -= __uint_as_float(w[i] & 0xffff0000u);
        }
    }
}

// Predicated loads, zero where the predicate is off: no branch, so nothing
// waits for a load before its value is split.
__device__ __forceinline__ void ld4_if(bool on, const float *p, float &a, float &b, float &c, float &d) {
    asm volatile("{.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                 "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
                 "@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%5];}"
                 : "=&f"(a), "=&f"(b), "=&f"(c), "=&f"(d)
                 : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void ld1_if(bool on, const float *p, float &a) {
    asm volatile("{.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\tmov.f32 %0, 0f00000000;\n\t@q ld.global.nc.f32 %0, [%2];}"
                 : "=&f"(a)
                 : "r"((int)on), "l"(p));
}

__device__ __forceinline__ void ld4(const float *p, float &a, float &b, float &c, float &d) {
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "l"(p));
}
__device__ __forceinline__ void ld1(const float *p, float &a) {
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(a) : "l"(p));
}

// Loads this lane's 8 elements of a unit.  p: the lane's first element of the
// slice; left: how much of K is left at the lane's first k (WHOLE: all of it).
// Rows past the operand's end are clamped by the caller: what they hold only
// reaches rows or columns of C that are not stored.  kAlongVec leaves out the
// last K % 4 elements (tail_unit).
template <int KIND, bool WHOLE>
__device__ __forceinline__ void load_unit(const float *p, int64_t ld, int rows, int left, float (&v)[8]) {
    if constexpr (KIND == kAlongVec) {
        if constexpr (WHOLE) {
            ld4(p, v[0], v[1], v[2], v[3]);
            ld4(p + 4, v[4], v[5], v[6], v[7]);
        } else {
            ld4_if(left >= 4, p, v[0], v[1], v[2], v[3]);
            ld4_if(left >= 8, p + 4, v[4], v[5], v[6], v[7]);
        }
    } else if constexpr (KIND == kAlong) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if constexpr (WHOLE) {
                ld1(p, v[2 * j]);
                ld1(p + 1, v[2 * j + 1]);
            } else {
                ld1_if(left > 0, p, v[2 * j]);
                ld1_if(left > 1, p + 1, v[2 * j + 1]);
            }
            if (j + 1 < rows) p += ld;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if constexpr (WHOLE) ld1(p, v[e]);
            else ld1_if(e < left, p, v[e]);
            p += ld;
        }
    }
}

// The elements past the last whole vector of a kAlongVec row (K % 4 of them,
// in the last slice only), read as they are needed.
__device__ __forceinline__ void tail_unit(const float *p, int left, float (&v)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e)
        if (e < left && e >= (left & ~3)) v[e] = __ldg(p + e);
}

template <int KIND, int NP>
__device__ __forceinline__ void store_unit(int u, int lane, const float (&v)[8], uint8_t *tile,
                                           uint32_t piece_bytes) {
    uint32_t w[4][NP];
#pragma unroll
    for (int j = 0; j < 4; ++j) split_pair<NP>(v[2 * j], v[2 * j + 1], w[j]);
    if constexpr (KIND == kAlong) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = u * 4 + j;
#pragma unroll
            for (int i = 0; i < NP; ++i)
                *reinterpret_cast<uint32_t *>(tile + i * piece_bytes + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) +
                                              (lane & 3) * 4) = w[j][i];
        }
    } else {
        const int r = KIND == kAlongVec ? u * 4 + (lane >> 3) : (u >> 3) * 32 + lane;
        const int c = KIND == kAlongVec ? (lane & 7) : (u & 7);
#pragma unroll
        for (int i = 0; i < NP; ++i)
            *reinterpret_cast<uint4 *>(tile + i * piece_bytes + r * 128 + ((c ^ (r & 7)) << 4)) =
                make_uint4(w[0][i], w[1][i], w[2][i], w[3][i]);
    }
}

template <int MODE, int AM, int BN_, int KA, int KB>
__global__ void __launch_bounds__(kThreads, 1) tc_gemm_direct_kernel(const __grid_constant__ Args a) {
    using L = Cfg<MODE, AM, BN_>;
    using MD = Mode<MODE>;
    constexpr int S = L::STAGES, NP = L::NP;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[S], empty[S], tfull[kBuffers], tempty[kBuffers], mma_done;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ int mma_aborted;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int64_t m0 = (int64_t)(blockIdx.x % a.tiles_m) * 128, n0 = (int64_t)(blockIdx.x / a.tiles_m) * BN_;
    const int64_t z = blockIdx.y;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], L::WPS);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < kBuffers; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], kWarps);
        }
        mbar_init(&mma_done, 1);
        fence_mbarrier_init();
        abort_flag = 0;
        mma_aborted = 0;
    }
    if (warp == kWarps) {
        tc::tmem_alloc(&tmem_base, kBuffers * BN_);
        tc::tmem_relinquish();
    }
    // rows past M or N are never stored by the units below: clear them once
    if (m0 + 128 > a.M || n0 + BN_ > a.N)
        for (uint32_t o = threadIdx.x * 16; o < S * L::STAGE; o += kThreads * 16)
            *reinterpret_cast<uint4 *>(smem + o) = make_uint4(0, 0, 0, 0);
    fence_proxy_async_shared();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const int nsl = a.nslices, seg = a.seg, K = (int)a.K;

    if (warp >= kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssuerRegs));
        if (warp == kWarps) {
            // ---- MMA issuer: the whole warp walks the slices, so that addresses
            // and descriptors stay warp-uniform, and one elected lane issues ----
            constexpr uint32_t idesc = tc::idesc_bf16_f32(128, BN_);
            const uint32_t ring = smem_u32(smem);
            const uint64_t desc0 = tc::smem_desc_kmajor(ring, 1024, tc::kSwizzle128B);
            int s = 0, b = 0, in_seg = 0;
            uint32_t ph = 0, bph = 1;
            bool stop = false;
            for (int i = 0; i < nsl; ++i) {
                const bool first = in_seg == 0;
                if (first && !tc::wait_warp(&tempty[b], bph, kWaitNs, &abort_flag)) stop = true;
                if (!stop && !tc::wait_warp(&full[s], ph, kWaitNs, &abort_flag)) stop = true;
                if (stop) {
                    if (lane == 0) {
                        if (!abort_flag) report_fault(a.fault, kFaultTcMmaWait);
                        abort_flag = 1;
                    }
                    break;
                }
                tc::fence_after_sync();
                const uint32_t d = tmem + (uint32_t)(b * BN_);
                const uint64_t at = desc0 + (uint64_t)(s * (L::STAGE >> 4));
                const uint64_t bt = at + ((NP * L::A_TILE) >> 4);
                const int ksteps = i == nsl - 1 ? a.last_ksteps : kSlice / 16;
                const bool last = ++in_seg == seg || i == nsl - 1;
                if (tc::elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kSlice / 16; ++kk) {
                        if (kk < 2 || ksteps > 2) {
#pragma unroll
                            for (int j = 0; j < MD::NPROD; ++j)
                                tc::mma_bf16(d, at + ((MD::pa(j) * L::A_TILE + kk * 32) >> 4),
                                             bt + ((MD::pb(j) * L::B_TILE + kk * 32) >> 4), idesc,
                                             (first && kk == 0 && j == 0) ? 0u : 1u);
                        }
                    }
                    tc::commit_to(&empty[s]);
                    if (last) tc::commit_to(&tfull[b]);
                }
                __syncwarp();
                if (last) {
                    in_seg = 0;
                    if (++b == kBuffers) {
                        b = 0;
                        bph ^= 1u;
                    }
                }
                if (++s == S) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (stop && tc::elect_one()) {
                mma_aborted = 1;
                tc::commit_to(&mma_done);
            }
        }
        __syncwarp();
    } else {
        // ---- load, split, promote ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWorkerRegs));
        // A slice is WPS warps' work and a warp takes every GROUPS-th one: its
        // loads fly while the other groups split.  (Several slices per warp in
        // flight did not overlap: waiting for the oldest waited for them all.)
        constexpr int JA = L::JA, U = L::JA + L::JB, G = L::GROUPS;
        const Source sa = a.a, sb = a.b;
        const int group = warp / L::WPS, wig = warp % L::WPS;
        const float *up[U];
        int rows[U];  // kAlong: how many of the unit's four rows exist
        bool live[U];
        auto place = [&](auto kind, int j, const Source &q, int64_t r0, int u) {
            constexpr int KIND = decltype(kind)::value;
            const int64_t first = r0 + (KIND == kAcross ? (u >> 3) * 32 : u * 4);
            const int64_t r = min(first + (KIND == kAlongVec ? (lane >> 3) : KIND == kAcross ? lane : 0), q.rows - 1);
            live[j] = first < q.rows;
            rows[j] = (int)min((int64_t)4, q.rows - r);
            const float *base = q.p + z * q.stride;
            if constexpr (KIND == kAcross) up[j] = base + (int64_t)(group * kSlice + (u & 7) * 8) * q.ld + r;
            else up[j] = base + r * q.ld + group * kSlice + (KIND == kAlongVec ? (lane & 7) * 8 : lane * 2);
        };
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (j < JA) place(Int<KA>(), j, sa, m0, wig + L::WPS * j);
            else place(Int<KB>(), j, sb, n0, wig + L::WPS * (j - JA));
        }
        // the lane's first k inside a slice
        auto lane_k = [&](int kind, int u) {
            return kind == kAlongVec ? (lane & 7) * 8 : kind == kAlong ? lane * 2 : (u & 7) * 8;
        };
        const int64_t step_a = G * (KA == kAcross ? kSlice * sa.ld : kSlice);
        const int64_t step_b = G * (KB == kAcross ? kSlice * sb.ld : kSlice);
        float x[U][8];
        auto load = [&](int i) {
            const int left = K - i * kSlice;
            if (left >= kSlice) {
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    if (!live[j]) continue;
                    if (j < JA) load_unit<KA, true>(up[j], sa.ld, rows[j], 0, x[j]);
                    else load_unit<KB, true>(up[j], sb.ld, rows[j], 0, x[j]);
                }
            } else if (left > 0) {
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    if (!live[j]) continue;
                    if (j < JA) load_unit<KA, false>(up[j], sa.ld, rows[j], left - lane_k(KA, wig + L::WPS * j), x[j]);
                    else load_unit<KB, false>(up[j], sb.ld, rows[j], left - lane_k(KB, wig + L::WPS * (j - JA)), x[j]);
                }
            }
        };
        const int quarter = warp & 3, part = warp >> 2;
        const uint32_t tcol = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * L::PC);
        float acc[L::PC];
#pragma unroll
        for (int c = 0; c < L::PC; ++c) acc[c] = 0.0f;
        int drained = 0;
        bool ok = true;
        auto drain = [&]() {
            const int b = drained % kBuffers;
            if (!tc::wait_warp(&tfull[b], (uint32_t)(drained / kBuffers) & 1u, 2 * kWaitNs, &abort_flag)) {
                if (!abort_flag) report_fault(a.fault, kFaultTcEpilogueWait);
                abort_flag = 1;
                ok = false;
                return;
            }
            __syncwarp();
            tc::fence_after_sync();
#pragma unroll
            for (int c = 0; c < L::PC; c += L::LD) {
                uint32_t r[L::LD];
                if constexpr (L::LD == 8) tc::tmem_ld_32x32b_x8(tcol + (uint32_t)(b * BN_ + c), r);
                else tc::tmem_ld_32x32b_x16(tcol + (uint32_t)(b * BN_ + c), r);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < L::LD; ++e) acc[c + e] = __fadd_rn(acc[c + e], __uint_as_float(r[e]));
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[b]);
            ++drained;
        };
        load(group);
        for (int i = group; i < nsl && ok; i += G) {
            const int s = i % S;
            // the MMAs this stage waits for may wait for a buffer of ours
            while (ok && (int64_t)(drained + kBuffers) * seg <= i - S) drain();
            if (!ok) break;
            if (!tc::wait_warp(&empty[s], ((uint32_t)(i / S) & 1u) ^ 1u, kWaitNs, &abort_flag)) {
                if (!abort_flag) report_fault(a.fault, kFaultTcProducerWait);
                abort_flag = 1;
                ok = false;
                break;
            }
            uint8_t *at = smem + s * L::STAGE, *bt = at + NP * L::A_TILE;
            if ((KA == kAlongVec || KB == kAlongVec) && i == nsl - 1 && (K & 3)) {
                const int left = K - i * kSlice;
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    if (!live[j]) continue;
                    if (KA == kAlongVec && j < JA) tail_unit(up[j], left - lane_k(KA, 0), x[j]);
                    if (KB == kAlongVec && j >= JA) tail_unit(up[j], left - lane_k(KB, 0), x[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < U; ++j) {
                if (!live[j]) continue;
                if (j < JA) store_unit<KA, NP>(wig + L::WPS * j, lane, x[j], at, L::A_TILE);
                else store_unit<KB, NP>(wig + L::WPS * (j - JA), lane, x[j], bt, L::B_TILE);
            }
            fence_proxy_async_shared();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
#pragma unroll
            for (int j = 0; j < U; ++j) up[j] += j < JA ? step_a : step_b;
            load(i + G);
            // this stage's previous MMAs are done, so every segment before them is
            while (ok && (int64_t)(drained + 1) * seg <= i - S) drain();
        }
        const int nseg = (nsl + seg - 1) / seg;
        while (ok && drained < nseg) drain();
        // ---- C through shared memory: every MMA has completed, the ring is free ----
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kWarps) : "memory");
        if (ok && !abort_flag) {
            float *ct = reinterpret_cast<float *>(smem);
#pragma unroll
            for (int c = 0; c < L::PC; ++c) ct[(quarter * 32 + lane) * L::PITCH + part * L::PC + c] = acc[c];
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kWarps) : "memory");
        if (ok && !abort_flag) {
            const float *ct = reinterpret_cast<const float *>(smem);
            float *C = a.C + z * a.stride_c;
            constexpr int RW = 128 / kWarps, CW = BN_ / 32;  // rows per warp, columns per lane
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const int lr = warp + r * kWarps;
                const int64_t gr = m0 + lr;
                if (gr >= a.M) continue;
                float *crow = C + gr * a.ldc + n0;
#pragma unroll
                for (int c = 0; c < CW; ++c) {
                    const int lc = c * 32 + lane;
                    if (n0 + lc >= a.N) continue;
                    float x = ct[lr * L::PITCH + lc];
                    if (a.gemm) x = __fmaf_rn(a.alpha, x, a.beta == 0.0f ? 0.0f : a.beta * crow[lc]);
                    crow[lc] = x;
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    // after an abort the MMAs issued before it complete before TMEM is freed
    if (threadIdx.x == 0 && abort_flag && mma_aborted) tc::wait_timed(&mma_done, 0, kWaitNs, nullptr);
    __syncthreads();
    tc::fence_after_sync();
    if (warp == kWarps) tc::tmem_dealloc(tmem, kBuffers * BN_);
}

template <int MODE, int AM, int BN_, int KA, int KB>
int launch(const Geometry &g, Args a, cudaStream_t stream) {
    using L = Cfg<MODE, AM, BN_>;
    auto kern = tc_gemm_direct_kernel<MODE, AM, BN_, KA, KB>;
    static std::atomic<uint64_t> configured{0};  // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM);
        if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "tc direct smem attribute: %s", cudaGetErrorString(e));
        configured.fetch_or(bit, std::memory_order_release);
    }
    a.tiles_m = (int)((g.M + 127) / 128);
    const int64_t tiles_n = (g.N + BN_ - 1) / BN_;
    const dim3 grid((unsigned)(a.tiles_m * tiles_n), (unsigned)g.batch);
    kern<<<grid, kThreads, L::SMEM, stream>>>(a);
    return check_launch("tc_gemm_direct_kernel");
}

using Launch = int (*)(const Geometry &, Args, cudaStream_t);

template <int MODE, int AM, int BN_>
int launch_kinds(const Geometry &g, const Args &a, cudaStream_t stream) {
    static const Launch table[3][3] = {
        {launch<MODE, AM, BN_, 0, 0>, launch<MODE, AM, BN_, 0, 1>, launch<MODE, AM, BN_, 0, 2>},
        {launch<MODE, AM, BN_, 1, 0>, launch<MODE, AM, BN_, 1, 1>, launch<MODE, AM, BN_, 1, 2>},
        {launch<MODE, AM, BN_, 2, 0>, launch<MODE, AM, BN_, 2, 1>, launch<MODE, AM, BN_, 2, 2>}};
    return table[a.a.kind][a.b.kind](g, a, stream);
}

template <int MODE>
int launch_width(int bn, const Geometry &g, const Args &a, cudaStream_t stream) {
    if (g.M <= 64) return launch_kinds<MODE, 64, 32>(g, a, stream);
    if (bn == 32) return launch_kinds<MODE, 128, 32>(g, a, stream);
    return launch_kinds<MODE, 128, 64>(g, a, stream);
}

Source source(const float *p, int64_t ld, int64_t rows, int64_t stride, int64_t batch, bool across) {
    Source s;
    s.p = p;
    s.ld = ld;
    s.rows = rows;
    s.stride = stride;
    s.kind = across ? kAcross
                    : (aligned16(p) && ld % 4 == 0 && (batch == 1 || stride % 4 == 0)) ? kAlongVec : kAlong;
    return s;
}

}  // namespace direct

// Microseconds of either way in each mode: launches and set-up, a wave of tiles
// beyond the first (two-pass: any wave), 64 k of a tile (64-row tiles of width 32,
// 128-row tiles of width 32 and of 64; two-pass 128 or, on pairs, 256 x 256), a MB
// of C by plain stores; the share that 64 k take longer where A or B is read in
// pairs or stored across k; the split pass in TB/s along and across k.  Least
// squares of the logarithms over 1500 random products (device time, B200); four
// in five of 900 others lie within 20 %.
struct Costs {
    double start, wave, slice[3], c_mb, a_pairs, a_across, b_pairs, b_across;
    double two_start, two_wave, two_slice, two_c_mb, split_along, split_across;
};
static const Costs kCosts[3] = {
    {6.5, 1.8, {0.32, 0.60, 0.73}, 0.73, 0.47, 0.28, 0.22, 0.11, 11.8, 2.4, 0.36, 0.39, 5.5, 4.8},
    {7.15, 2.3, {0.44, 0.71, 0.91}, 0.71, 0.49, 0.27, 0.18, 0.06, 15.0, 1.2, 0.90, 0.38, 6.3, 5.1},
    {7.1, 2.2, {0.64, 0.96, 1.27}, 0.76, 0.28, 0.14, 0.16, 0.09, 14.3, 0.7, 1.93, 0.36, 5.9, 5.1}};

// Tile width of the one-launch contraction for a product, 0 where the
// two-pass path serves it: whichever of the two is estimated faster, the one
// launch by 8 % at least.  Over the 2400 products that loses 0.6 % against the
// better of the two each time.  Either side of the line, direct against two-pass:
// 64 x 4096 x 8192 BF16 56 and 86 us, split3 69 and 200, split6 100 and 351; 1024^3
// split3 21 and 27, BF16 18 and 16; 512^3 BF16 9.5 and 12.8; 1000 x 777 x 1100 BF16 18
// and 22; 1536^3 split3 54 and 37; 2000 x 2000 x 100 BF16 24 and 13; seven of 16 x 3688
// x 3320 BF16 183 and 133, of 31 x 1782 x 1419 split6 71 and 111.
int direct_width(const gatlas_matmul_desc *d, const Geometry &g, const float *A, const float *B, const float *C) {
    using namespace direct;
    if (d->engine == GATLAS_ENGINE_TC_FP8) return 0;  // block scales need whole 128 x 128 blocks first
    // split6 counts promotion intervals in slices of 32, two to a slice here
    if (d->engine == GATLAS_ENGINE_TC_SPLIT6 && d->extra % 2 != 0) return 0;
    if (g.M > (1 << 20) || g.N > (1 << 20) || g.K > (1 << 24)) return 0;
    // K beyond the transposing split's grid stays refused there
    if ((g.ta || !g.tb) && g.K > 65535 * 64) return 0;
    const int mode = d->engine == GATLAS_ENGINE_TC_BF16 ? 0 : d->engine == GATLAS_ENGINE_TC_SPLIT3 ? 1 : 2;
    const Costs &c = kCosts[mode];
    const double sms = sm_count(), slices = (double)((g.K + kSlice - 1) / kSlice), batch = (double)g.batch;
    const auto waves = [&](int64_t m, int64_t n, double units) {
        return std::ceil((double)((g.M + m - 1) / m) * (double)((g.N + n - 1) / n) * batch / units);
    };
    const int ka = source(A, g.lda, g.M, g.stride_a, g.batch, g.ta).kind;
    const int kb = source(B, g.ldb, g.N, g.stride_b, g.batch, !g.tb).kind;
    const bool reads_c = d->gemm && d->beta != 0.0;
    const double c_mb = batch * (double)g.M * (double)g.N * 4e-6 * (reads_c ? 2 : 1);
    const double slower = 1.0 + (ka == kAlong ? c.a_pairs : ka == kAcross ? c.a_across : 0.0) +
                          (kb == kAlong ? c.b_pairs : kb == kAcross ? c.b_across : 0.0);
    const auto direct_us = [&](int bn) {
        const double w = waves(128, bn, sms);
        return c.start + w * slices * c.slice[g.M <= 64 ? 0 : bn == 32 ? 1 : 2] * slower + (w - 1) * c.wave + c_mb * c.c_mb;
    };
    const bool pair = mode != 0 && g.M > BM;
    const bool plain_c = reads_c || g.ldc % 4 != 0 || !aligned16(C) || (g.batch > 1 && g.stride_c % 4 != 0);
    const double w2 = waves(pair ? 256 : 128, 256, pair ? sms / 2 : sms);
    const double mb_per_row = batch * (double)g.K * (4 + 2 * (mode + 1)) * 1e-6;
    const double split_us = mb_per_row * ((double)g.M / (g.ta ? c.split_across : c.split_along) +
                                          (double)g.N / (g.tb ? c.split_along : c.split_across));
    const double two_pass_us =
        c.two_start + split_us + w2 * (slices * c.two_slice + c.two_wave) + (plain_c ? c_mb * c.two_c_mb : 0.0);
    const double us32 = direct_us(32), us64 = g.M <= 64 ? us32 : direct_us(64);
    if (std::min(us32, us64) * 1.08 > two_pass_us) return 0;
    return us32 <= us64 ? 32 : 64;
}

int matmul_direct(const gatlas_matmul_desc *d, const Geometry &g, int bn, const float *A, const float *B, float *C,
                  cudaStream_t stream) {
    using namespace direct;
    const int mode = d->engine == GATLAS_ENGINE_TC_BF16 ? 0 : d->engine == GATLAS_ENGINE_TC_SPLIT3 ? 1 : 2;
    Args a;
    std::memset(&a, 0, sizeof(a));
    a.a = source(A, g.lda, g.M, g.stride_a, g.batch, g.ta);
    a.b = source(B, g.ldb, g.N, g.stride_b, g.batch, !g.tb);
    a.C = C;
    a.M = g.M, a.N = g.N, a.K = g.K, a.ldc = g.ldc, a.stride_c = g.stride_c;
    a.nslices = (int)((g.K + kSlice - 1) / kSlice);
    // (split6 counts slices of 32; its interval here is even)
    a.seg = mode == 2 ? promotion_interval(d->extra, mode, 2 * a.nslices) / 2
                      : promotion_interval(d->extra, mode, a.nslices);
    // the two-pass path stages split6 in slices of 32: half a slice of steps where the second half is empty
    a.last_ksteps = mode == 2 && g.K - (int64_t)(a.nslices - 1) * kSlice <= 32 ? 2 : kSlice / 16;
    a.alpha = (float)d->alpha, a.beta = (float)d->beta, a.gemm = d->gemm;
    a.fault = device_fault_word();
    switch (mode) {
        case 0: return launch_width<0>(bn, g, a, stream);
        case 1: return launch_width<1>(bn, g, a, stream);
        default: return launch_width<2>(bn, g, a, stream);
    }
}

}  // namespace tcg
}  // namespace gatlas
