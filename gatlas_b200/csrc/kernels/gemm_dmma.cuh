// Double-precision GEMM on the FP64 tensor-core instruction (mma.sync
// m16n8k4.f64), the buffer engine's default point for double.
//
// Arithmetic: the instruction adds its four products to each accumulator as
// fused multiply-adds in k order, each rounded to nearest, so a chain of them
// over k = 0..K-1 gives the reference's mad chain (KernelMatmulBuffer.hpp:
// 302-321) bit for bit, as the SIMT kernel does.  The tests compare it with
// the sequential fma chain, signed zeros and infinities included.
//
// What bounds it: the FP64 pipe, 64 multiply-adds per SM and cycle (37.1
// TFLOP/s measured for the bare instruction, 34.1 for scalar fma).  The scalar
// kernel (8 x 16 threads of 8 x 8) sits at two warps per scheduler and spends
// 16 instructions of shared-memory traffic and issue where this one spends
// two loads and one instruction per 512 multiply-adds.  Measured: 4096 x 4096 x
// 2048 at 33.4 TFLOP/s (scalar kernel 21.0), 1531 x 1277 x 1021 with odd
// leading dimensions in 153 us (657).
//
// Layout: a K step of 16 lands in shared memory by asynchronous copies in the
// operand's own order, with no transposition and no staging registers: rows
// of 16 k (pitch 20) for an operand stored along k, rows of the tile's m or n
// (pitch tile + 4) for one stored across it.  Either pitch is 4 modulo 16
// doubles, so the fragment reads (8 rows x 4 k per warp) touch every bank
// once.  Copies are 16 bytes wide where base, leading dimension and instance
// stride allow it and 8 bytes otherwise, so odd leading dimensions keep the
// same kernel; elements past M, N and K are zero-filled by the copies.
#pragma once

#include "../common.cuh"

namespace gatlas {
namespace dmma {

struct Args {
    const double *A, *B;
    double *C;
    int64_t M, N, K, lda, ldb, ldc, stride_a, stride_b, stride_c;
    double alpha, beta;
    int gemm;
    int vec_a, vec_b;  // 16-byte copies allowed
    int tiles_m, tiles_n;
};

constexpr int BK = 16;
constexpr int kStages = 4;
constexpr int kGroup = 8;  // tile rows per raster group: neighbouring CTAs share A and B rows in L2

template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, uint32_t bytes) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes)
                     : "memory");
}

__device__ __forceinline__ void mma_m16n8k4(double (&c)[4], const double (&a)[2], double b) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(b));
}

// One operand's part of a stage: R rows of the tile (m or n) by BK.  KMAJOR:
// stored along k ([R][BK], pitch BK + 4); otherwise [BK][R], pitch R + 4.
template <int R, bool KMAJOR>
struct Operand {
    static constexpr int PITCH = KMAJOR ? BK + 4 : R + 4;
    static constexpr int ELEMS = KMAJOR ? R * PITCH : BK * PITCH;
    __device__ static __forceinline__ int at(int r, int k) { return KMAJOR ? r * PITCH + k : k * PITCH + r; }
};

// A thread's share of an operand's copies, W doubles (8 or 16 bytes) each:
// one place along the contiguous dimension and every STEP-th row across it,
// so that a K step costs one pointer addition and one comparison per copy.
template <int R, bool KMAJOR, int NT, int W>
struct Loader {
    using O = Operand<R, KMAJOR>;
    static constexpr int OUTER = KMAJOR ? R : BK, INNER = KMAJOR ? BK : R;
    static constexpr int PER_ROW = INNER / W, STEP = NT / PER_ROW;
    static constexpr int COPIES = (OUTER + STEP - 1) / STEP;
    static_assert(NT % PER_ROW == 0, "a thread keeps its place along the row");

    // Copies tile rows [r0, r0 + R) (m or n, of `rows`) and k [k0, k0 + BK).
    __device__ static __forceinline__ void copy(double *smem, const double *src, int64_t ld, int64_t r0, int64_t rows,
                                                int64_t k0, int64_t K, int tid) {
        const int o = tid / PER_ROW, i = tid % PER_ROW * W;
        const int64_t go = (KMAJOR ? r0 : k0) + o, gi = (KMAJOR ? k0 : r0) + i;
        const int64_t oleft = (KMAJOR ? rows : K) - go, ileft = (KMAJOR ? K : rows) - gi;
        const uint32_t bytes = ileft >= W ? W * 8u : (ileft > 0 ? (uint32_t)ileft * 8u : 0u);
        const double *p = src + go * ld + gi;
        double *d = smem + o * O::PITCH + i;
#pragma unroll
        for (int j = 0; j < COPIES; ++j) {
            if (OUTER % STEP == 0 || o + j * STEP < OUTER) {
                const uint32_t n = j * STEP < oleft ? bytes : 0u;
                cp_async<W * 8>(d + j * STEP * O::PITCH, n ? p : src, n);
            }
            p += (int64_t)STEP * ld;
        }
    }
};

template <int R, bool KMAJOR, int NT>
__device__ __forceinline__ void load_operand(double *smem, const double *src, int64_t ld, int64_t r0, int64_t rows,
                                             int64_t k0, int64_t K, bool vec, int tid) {
    if (vec) Loader<R, KMAJOR, NT, 2>::copy(smem, src, ld, r0, rows, k0, K, tid);
    else Loader<R, KMAJOR, NT, 1>::copy(smem, src, ld, r0, rows, k0, K, tid);
}

template <int BM, int BN, bool TA, bool TB>
constexpr int stage_elems() {
    return Operand<BM, !TA>::ELEMS + Operand<BN, TB>::ELEMS;
}
template <int BM, int BN, bool TA, bool TB>
constexpr int smem_bytes() {
    return kStages * stage_elems<BM, BN, TA, TB>() * (int)sizeof(double);
}

// BM x BN tile of C per CTA, WM x WN per warp.
template <int BM, int BN, int WM, int WN, bool TA, bool TB>
__global__ void __launch_bounds__(BM / WM *(BN / WN) * 32, BM *BN >= 64 * 32 ? 3 : 4) gemm_dmma_kernel(Args a) {
    constexpr int NT = BM / WM * (BN / WN) * 32;
    constexpr int MI = WM / 16, NI = WN / 8;
    using OA = Operand<BM, !TA>;
    using OB = Operand<BN, TB>;
    constexpr int STAGE = stage_elems<BM, BN, TA, TB>();
    extern __shared__ __align__(16) double dmma_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = warp / (BN / WN) * WM, wn = warp % (BN / WN) * WN;
    // grouped raster: tile rows in groups of kGroup, tile columns within a group
    const int per_group = kGroup * a.tiles_n;
    const int first = (int)(blockIdx.x / per_group) * kGroup;
    const int gm = min(a.tiles_m - first, kGroup);
    const int rem = (int)(blockIdx.x % per_group);
    const int64_t m0 = (int64_t)(first + rem % gm) * BM, n0 = (int64_t)(rem / gm) * BN;
    const double *A = a.A + (int64_t)blockIdx.z * a.stride_a;
    const double *B = a.B + (int64_t)blockIdx.z * a.stride_b;

    auto issue = [&](int64_t kt) {
        double *s = dmma_smem + (int)(kt % kStages) * STAGE;
        load_operand<BM, !TA, NT>(s, A, a.lda, m0, a.M, kt * BK, a.K, a.vec_a, tid);
        load_operand<BN, TB, NT>(s + OA::ELEMS, B, a.ldb, n0, a.N, kt * BK, a.K, a.vec_b, tid);
    };
    const int64_t KT = (a.K + BK - 1) / BK;
    for (int64_t kt = 0; kt < kStages - 1; ++kt) {
        if (kt < KT) issue(kt);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    double acc[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

    for (int64_t kt = 0; kt < KT; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // step kt has landed for every thread, and step kt - 1 is read
        const double *as = dmma_smem + (int)(kt % kStages) * STAGE;
        const double *bs = as + OA::ELEMS;
        double af[2][MI][2], bf[2][NI];
        auto fragments = [&](int b, int k4) {
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                af[b][i][0] = as[OA::at(wm + i * 16 + g, k4 + t)];
                af[b][i][1] = as[OA::at(wm + i * 16 + 8 + g, k4 + t)];
            }
#pragma unroll
            for (int j = 0; j < NI; ++j) bf[b][j] = bs[OB::at(wn + j * 8 + g, k4 + t)];
        };
        fragments(0, 0);
#pragma unroll
        for (int q = 0; q < BK / 4; ++q) {
            // the next four k's fragments load behind this four's multiply-adds,
            // and the copies of a later step issue behind the first four's
            if (q + 1 < BK / 4) fragments((q + 1) & 1, 4 * (q + 1));
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NI; ++j) mma_m16n8k4(acc[i][j], af[q & 1][i], bf[q & 1][j]);
            if (q == 0) {
                if (kt + kStages - 1 < KT) issue(kt + kStages - 1);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    double *C = a.C + (int64_t)blockIdx.z * a.stride_c;
    const bool reads_c = a.gemm && a.beta != 0.0;
    // 16 rows of C at a time, all their reads in flight together (one at a time,
    // 2048 x 2048 x 64 with beta = 0.5 ran 40 us, so 31); 16-byte
    // accesses where every pair of columns of the tile is whole.
    const bool vec_c =
        a.ldc % 2 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (a.N % 2 == 0 || n0 + BN <= a.N);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        double old[2][NI][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t row = m0 + wm + i * 16 + h * 8 + g;
            const double *crow = C + row * a.ldc;
#pragma unroll
            for (int j = 0; j < NI; ++j) {
                const int64_t col = n0 + wn + j * 8 + 2 * t;
                old[h][j][0] = old[h][j][1] = 0.0;
                if (!reads_c) continue;
                if (vec_c) {
                    if (row < a.M && col < a.N) {
                        const double2 v = *reinterpret_cast<const double2 *>(crow + col);
                        old[h][j][0] = v.x, old[h][j][1] = v.y;
                    }
                } else {
                    if (row < a.M && col < a.N) old[h][j][0] = crow[col];
                    if (row < a.M && col + 1 < a.N) old[h][j][1] = crow[col + 1];
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t row = m0 + wm + i * 16 + h * 8 + g;
            double *crow = C + row * a.ldc;
#pragma unroll
            for (int j = 0; j < NI; ++j) {
                const int64_t col = n0 + wn + j * 8 + 2 * t;
                double v[2] = {acc[i][j][2 * h], acc[i][j][2 * h + 1]};
                if (a.gemm) {
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        v[e] = __fma_rn(a.alpha, v[e], reads_c ? a.beta * old[h][j][e] : 0.0);
                }
                if (vec_c) {
                    if (row < a.M && col < a.N) *reinterpret_cast<double2 *>(crow + col) = make_double2(v[0], v[1]);
                } else {
                    if (row < a.M && col < a.N) crow[col] = v[0];
                    if (row < a.M && col + 1 < a.N) crow[col + 1] = v[1];
                }
            }
        }
    }
}

}  // namespace dmma
}  // namespace gatlas
