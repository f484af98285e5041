// Single-precision SIMT GEMM of the buffer engine's default point.
//
// Arithmetic: one fused multiply-add chain per element over k = 0..K-1, two
// neighbouring columns per packed instruction (fma.rn.f32x2), bit-exact
// against a sequential fmaf chain like every SIMT point (gemm_simt.cuh).
//
// What bounds it: at large sizes the FP32 pipe and shared-memory reads together
// (8 x 8 per thread reads 50 cycles of shared memory per 64 of multiply-adds,
// 8 x 16 per thread 75 per 128), at small ones how many warps an SM has to
// hide latency with, so the tile follows the size (gemm_ffma.cu).
//
// Against the register-staged kernel of the explicit points: operands land by
// asynchronous copies, 3 or 4 steps of 16 k in flight, in the order they are
// stored in, 16 bytes wide where base, leading dimension and instance stride
// allow and 4 otherwise; no staging registers (so 8 x 16 fits without spills)
// and no transposing stores.  A stored along k is read from its own rows, four
// k at a time.  B stored along k is turned once in shared memory, a step ahead,
// because packed multiply-adds need neighbouring columns in neighbouring
// registers (packing them by moves instead ran 29 TFLOP/s, scalar
// multiply-adds 37, turning 43 at 3072 x 2560 x 2048).
//
// The epilogue reads C a batch of rows at a time (element by element, each
// waited for, a product of 3584 x 3072 x 64 with beta = 0.5 ran 62 us, in
// batches 42; 1024^3 66 -> 62, 2047 x 2049 x 255 80 -> 68).
//
// Measured, default point before and after: 1024^3 119 -> 62 us, 256^3 36 -> 8,
// 1001 x 1003 x 999 190 -> 69, 3072 x 2560 x 2048 with B transposed 896 -> 752,
// 8192 x 8192 x 2048 50.3 -> 54.2 TFLOP/s.
#pragma once

#include <type_traits>

#include "../common.cuh"

namespace gatlas {
namespace ffma {

struct Args {
    const float *A, *B;
    float *C;
    int64_t M, N, K, lda, ldb, ldc, stride_a, stride_b, stride_c;
    float alpha, beta;
    int gemm;
    int vec_a, vec_b;  // 16-byte copies allowed
    int tiles_m, tiles_n;
};

constexpr int BK = 16;
constexpr int kGroup = 8;  // tile rows per raster group: neighbouring CTAs share A and B rows in L2

template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, uint32_t bytes) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes)
                     : "memory");
}

// d0 = a*b0 + d0, d1 = a*b1 + d1, each a round-to-nearest fused multiply-add
__device__ __forceinline__ void fma2(float &d0, float &d1, float a, float b0, float b1) {
    asm("{.reg .b64 pa, pb, pd;\n\t"
        "mov.b64 pa, {%2, %2};\n\t"
        "mov.b64 pb, {%3, %4};\n\t"
        "mov.b64 pd, {%0, %1};\n\t"
        "fma.rn.f32x2 pd, pa, pb, pd;\n\t"
        "mov.b64 {%0, %1}, pd;}"
        : "+f"(d0), "+f"(d1)
        : "f"(a), "f"(b0), "f"(b1));
}

// One operand's part of a stage.  KMAJOR (stored along k): [R][BK], pitch
// BK + 4, so that 16-byte reads of neighbouring rows fall in distinct banks;
// otherwise [BK][R].
template <int R, bool KMAJOR>
struct Operand {
    static constexpr int PITCH = KMAJOR ? BK + 4 : R;
    static constexpr int ELEMS = KMAJOR ? R * PITCH : BK * PITCH;
};

// A thread's share of an operand's copies, W floats each: one place along the
// contiguous dimension and every STEP-th row across it.
template <int R, bool KMAJOR, int NT, int W>
struct Loader {
    using O = Operand<R, KMAJOR>;
    static constexpr int OUTER = KMAJOR ? R : BK, INNER = KMAJOR ? BK : R;
    static constexpr int PER_ROW = INNER / W;
    static constexpr int COPIES = (OUTER * PER_ROW + NT - 1) / NT;

    __device__ static __forceinline__ void copy(float *smem, const float *src, int64_t ld, int64_t r0, int64_t rows,
                                                int64_t k0, int64_t K, int tid) {
        const int64_t obase = KMAJOR ? r0 : k0, ibase = KMAJOR ? k0 : r0;
        const int64_t olim = KMAJOR ? rows : K, ilim = KMAJOR ? K : rows;
        if constexpr (NT % PER_ROW == 0) {
            constexpr int STEP = NT / PER_ROW;
            const int o = tid / PER_ROW, i = tid % PER_ROW * W;
            const int64_t oleft = olim - obase - o, ileft = ilim - ibase - i;
            const uint32_t bytes = ileft >= W ? W * 4u : (ileft > 0 ? (uint32_t)ileft * 4u : 0u);
            const float *p = src + (obase + o) * ld + ibase + i;
            float *d = smem + o * O::PITCH + i;
#pragma unroll
            for (int j = 0; j < COPIES; ++j) {
                if (OUTER % STEP == 0 || o + j * STEP < OUTER) {
                    const uint32_t n = j * STEP < oleft ? bytes : 0u;
                    cp_async<W * 4>(d + j * STEP * O::PITCH, n ? p : src, n);
                }
                p += (int64_t)STEP * ld;
            }
        } else {  // rows wider than the thread block: NT places along one row at a time
            static_assert(PER_ROW % NT == 0, "copies divide among the threads");
            constexpr int PARTS = PER_ROW / NT;
#pragma unroll
            for (int j = 0; j < COPIES; ++j) {
                const int o = j / PARTS, i = (j % PARTS * NT + tid) * W;
                const int64_t ileft = ilim - ibase - i;
                const uint32_t bytes = ileft >= W ? W * 4u : (ileft > 0 ? (uint32_t)ileft * 4u : 0u);
                const uint32_t n = obase + o < olim ? bytes : 0u;
                cp_async<W * 4>(smem + o * O::PITCH + i, n ? src + (obase + o) * ld + ibase + i : src, n);
            }
        }
    }
};

template <int R, bool KMAJOR, int NT>
__device__ __forceinline__ void load_operand(float *smem, const float *src, int64_t ld, int64_t r0, int64_t rows,
                                             int64_t k0, int64_t K, bool vec, int tid) {
    if (vec) Loader<R, KMAJOR, NT, 4>::copy(smem, src, ld, r0, rows, k0, K, tid);
    else Loader<R, KMAJOR, NT, 1>::copy(smem, src, ld, r0, rows, k0, K, tid);
}

// Index inside the warp tile of micro-tile element i of lane coordinate l
// (of L): neighbouring lanes take neighbouring rows of a k-major tile, and
// neighbouring groups of four of one stored across k.
template <bool KMAJOR, int L>
__device__ __forceinline__ int micro(int l, int i) {
    return KMAJOR ? i * L + l : (i / 4) * (L * 4) + l * 4 + (i & 3);
}

// Fragments of four k: f[q][i] = element i at k0 + q.
template <int R, bool KMAJOR, int L, int T>
__device__ __forceinline__ void fragment(const float *s, int base, int l, int k0, float (&f)[4][T]) {
    using O = Operand<R, KMAJOR>;
    if constexpr (KMAJOR) {
#pragma unroll
        for (int i = 0; i < T; ++i) {
            const float4 v = *reinterpret_cast<const float4 *>(s + (base + micro<true, L>(l, i)) * O::PITCH + k0);
            f[0][i] = v.x, f[1][i] = v.y, f[2][i] = v.z, f[3][i] = v.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < T; i += 4) {
                const float4 v = *reinterpret_cast<const float4 *>(s + (k0 + q) * O::PITCH + base + micro<false, L>(l, i));
                f[q][i] = v.x, f[q][i + 1] = v.y, f[q][i + 2] = v.z, f[q][i + 3] = v.w;
            }
    }
}

// Turns a k-major tile [R][BK] (pitch BK + 4) into [BK][R]: a warp reads one
// 16-byte run of k of 32 neighbouring rows and writes four rows of k, both
// without bank conflicts.
template <int R, int NT>
__device__ __forceinline__ void transpose_tile(const float *src, float *dst, int tid) {
#pragma unroll
    for (int e = tid; e < R * (BK / 4); e += NT) {
        const int r = e % R, k = e / R * 4;
        const float4 v = *reinterpret_cast<const float4 *>(src + r * (BK + 4) + k);
        dst[k * R + r] = v.x, dst[(k + 1) * R + r] = v.y, dst[(k + 2) * R + r] = v.z, dst[(k + 3) * R + r] = v.w;
    }
}

// BM x BN tile of C per CTA, TM x TN per thread, LM lanes of a warp along m.
// AHEAD: a step's first fragments load during the previous step.
template <int BM, int BN, int TM, int TN, int LM, bool TA, bool TB, int STAGES, int MINB, bool AHEAD>
__global__ void __launch_bounds__(BM / TM *(BN / TN), MINB) gemm_ffma_kernel(Args a) {
    constexpr int NT = BM / TM * (BN / TN), LN = 32 / LM;
    constexpr int WM = LM * TM, WN = LN * TN;  // warp tile
    using OA = Operand<BM, !TA>;
    using OB = Operand<BN, TB>;
    constexpr int STAGE = OA::ELEMS + OB::ELEMS;
    extern __shared__ __align__(16) float ffma_smem[];
    float *turned = ffma_smem + STAGES * STAGE;  // TB: two steps of B as [BK][BN]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ly = lane / LN, lx = lane % LN;
    const int wm = warp / (BN / WN) * WM, wn = warp % (BN / WN) * WN;
    // grouped raster: tile rows in groups of kGroup, tile columns within a group
    const int per_group = kGroup * a.tiles_n;
    const int first = (int)(blockIdx.x / per_group) * kGroup;
    const int gm = min(a.tiles_m - first, kGroup);
    const int rem = (int)(blockIdx.x % per_group);
    const int64_t m0 = (int64_t)(first + rem % gm) * BM, n0 = (int64_t)(rem / gm) * BN;
    const float *A = a.A + (int64_t)blockIdx.z * a.stride_a;
    const float *B = a.B + (int64_t)blockIdx.z * a.stride_b;

    const int KT = (int)((a.K + BK - 1) / BK);
    auto stage = [&](int kt) { return ffma_smem + kt % STAGES * STAGE; };
    auto issue = [&](int kt) {
        if (kt < KT) {
            float *s = stage(kt);
            load_operand<BM, !TA, NT>(s, A, a.lda, m0, a.M, (int64_t)kt * BK, a.K, a.vec_a, tid);
            load_operand<BN, TB, NT>(s + OA::ELEMS, B, a.ldb, n0, a.N, (int64_t)kt * BK, a.K, a.vec_b, tid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto turn = [&](int kt) {  // step kt of B into its [BK][BN] buffer
        if (TB && kt < KT) transpose_tile<BN, NT>(stage(kt) + OA::ELEMS, turned + (kt & 1) * (BK * BN), tid);
    };
    // Steps that must have landed when step kt starts: kt itself, and kt + 1
    // where its B is turned during step kt.
    constexpr int PENDING = STAGES - 2 - (TB ? 1 : 0);
    static_assert(PENDING >= 0, "ring depth");
    auto arrive = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
        __syncthreads();
    };
    for (int kt = 0; kt < STAGES - 1; ++kt) issue(kt);

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    float af[2][4][TM], bf[2][4][TN];
    auto fragments = [&](int kt, int c, int b) {
        const float *s = stage(kt);
        fragment<BM, !TA, LM, TM>(s, wm, ly, 4 * c, af[b]);
        fragment<BN, false, LN, TN>(TB ? turned + (kt & 1) * (BK * BN) : s + OA::ELEMS, wn, lx, 4 * c, bf[b]);
    };
    arrive();
    if (TB) {
        turn(0);
        __syncthreads();
    }
    if (AHEAD && KT > 0) fragments(0, 0, 0);
    for (int kt = 0; kt < KT; ++kt) {
        if (!AHEAD) fragments(kt, 0, 0);
#pragma unroll
        for (int c = 0; c < BK / 4; ++c) {
            // the next four k's fragments load behind this four's multiply-adds
            if (c + 1 < BK / 4) {
                fragments(kt, c + 1, (c + 1) & 1);
            } else if (AHEAD) {
                arrive();  // step kt + 1 has landed for every thread, and step kt is read
                if (kt + 1 < KT) fragments(kt + 1, 0, 0);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; j += 2)
                        fma2(acc[i][j], acc[i][j + 1], af[c & 1][q][i], bf[c & 1][q][j], bf[c & 1][q][j + 1]);
            if (c == 0) {  // behind the first four's multiply-adds: later steps' copies, the next step's turn
                issue(kt + STAGES - 1);
                turn(kt + 1);
            }
        }
        if (!AHEAD) arrive();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    float *C = a.C + (int64_t)blockIdx.z * a.stride_c;
    const bool reads_c = a.gemm && a.beta != 0.0f;
    // Rows of C in batches of 32 elements a thread, all of a batch's reads in
    // flight together; 16-byte accesses where every group of four columns of the
    // tile is whole.
    const bool vec_c =
        a.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (a.N % 4 == 0 || n0 + BN <= a.N);
    float *Ct = C + m0 * a.ldc + n0;
    const int mleft = (int)min(a.M - m0, (int64_t)BM), nleft = (int)min(a.N - n0, (int64_t)BN);
    auto finish = [&](auto reads) {
        constexpr bool READS = decltype(reads)::value;
        constexpr int ROWS = TM < 32 / TN ? TM : 32 / TN;
#pragma unroll
        for (int i0 = 0; i0 < TM; i0 += ROWS) {
            float old[ROWS][TN];
            if constexpr (READS) {
#pragma unroll
                for (int i = 0; i < ROWS; ++i) {
                    const int row = wm + micro<!TA, LM>(ly, i0 + i);
                    const float *crow = Ct + row * a.ldc;
#pragma unroll
                    for (int j = 0; j < TN; j += 4) {
                        const int col = wn + micro<false, LN>(lx, j);
                        if (vec_c) {
                            if (row < mleft && col < nleft) {
                                const float4 v = *reinterpret_cast<const float4 *>(crow + col);
                                old[i][j] = v.x, old[i][j + 1] = v.y, old[i][j + 2] = v.z, old[i][j + 3] = v.w;
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (row < mleft && col + e < nleft) old[i][j + e] = crow[col + e];
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int row = wm + micro<!TA, LM>(ly, i0 + i);
                float *crow = Ct + row * a.ldc;
#pragma unroll
                for (int j = 0; j < TN; j += 4) {
                    const int col = wn + micro<false, LN>(lx, j);
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        v[e] = acc[i0 + i][j + e];
                        if (a.gemm) v[e] = __fmaf_rn(a.alpha, v[e], READS ? a.beta * old[i][j + e] : 0.0f);
                    }
                    if (vec_c) {
                        if (row < mleft && col < nleft)
                            *reinterpret_cast<float4 *>(crow + col) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (row < mleft && col + e < nleft) crow[col + e] = v[e];
                    }
                }
            }
        }
    };
    if (reads_c) finish(std::true_type{});
    else finish(std::false_type{});
}

template <int BM, int BN, bool TA, bool TB, int STAGES>
constexpr int smem_bytes() {
    return (STAGES * (Operand<BM, !TA>::ELEMS + Operand<BN, TB>::ELEMS) + (TB ? 2 * BK * BN : 0)) * (int)sizeof(float);
}

}  // namespace ffma
}  // namespace gatlas
