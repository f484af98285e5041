// Column-major GEMV (y = A^T-stored product) with the row segments of a column
// block summed inside a thread-block cluster.
//
// A CTA owns W columns and one segment of the rows; its 8 warps take
// interleaved groups of rows, 32 / LPR rows at a time with LPR lanes across the
// columns, CPL columns a lane (one 16-byte vector where rows are 16-byte
// aligned, else CPL coalesced 4- or 8-byte loads).  The partial sums of a
// block's segments, one CTA of a cluster each, are added in segment order by
// the first CTA over distributed shared memory: no partial sums in global
// memory, no arrival counters to clear and no second launch.
//
// Rounding: floats are summed U rows from zero, then added to the column's
// total, doubles into two accumulators (floats off the 16-byte grid with 8 rows
// in flight need neither), and a block's 8 warps add up in pairs, so that the
// sums are no longer than the general kernel's, whose 4 CTAs per SM cut the rows
// finer (one chain per lane: error against 64 bits at 16384^2 floats 1.56 times
// the general kernel's, at 20000 x 6000 1.3; now half).
//
// How many loads the compiler keeps in flight follows from what else holds
// registers, hence an instantiation's accumulators and CTAs per SM: doubles with
// two accumulators 116 us at 3396 x 27644, with one 128, with sums from zero 146.
#pragma once

#include <string.h>

#include "../common.cuh"
#include "../tcgen05.cuh"

namespace gatlas {
namespace gvc {

struct Args {
    const void *A, *x;
    void *y;
    size_t M, N, lda;
    size_t stride_a, stride_x, stride_y;
    double alpha, beta;
    int gemv;
    size_t seg_len;  // rows per segment; segment s of the cluster starts at s * seg_len
};

constexpr int kThreads = 256, kWarps = 8;

__device__ __forceinline__ float madd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double madd(double a, double b, double c) { return __fma_rn(a, b, c); }

__device__ __forceinline__ float ld_peer(uint32_t addr, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ double ld_peer(uint32_t addr, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}

// Streaming loads that stay where they are written: left to itself the
// compiler pairs loads with their multiply-adds to save registers, and half as
// many are in flight.
__device__ __forceinline__ void load_vec(const float *p, float (&v)[4]) {
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
}
__device__ __forceinline__ void load_vec(const double *p, double (&v)[2]) {
    asm volatile("ld.global.cs.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
}
__device__ __forceinline__ void load_one(const float *p, float &v) {
    asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p));
}
__device__ __forceinline__ void load_one(const double *p, double &v) {
    asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(v) : "l"(p));
}

// T; VEC: 16-byte loads (CPL = 16 / sizeof(T)); LPR lanes per row; U row groups in
// flight; SETS accumulators per column, rows dealt out among them, or 0: one, added
// to the column's total after every U rows; MINB CTAs per SM asked for (0: none)
template <typename T, bool VEC, int LPR, int CPL, int U, int SETS, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) gemv_cols_cluster_kernel(Args a) {
    constexpr int W = LPR * CPL, RPW = 32 / LPR;  // columns per block, rows per warp and group
    __shared__ T red[kWarps][W];
    __shared__ T sums[W];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int lc = lane % LPR, lr = lane / LPR;
    const size_t seg = blockIdx.y, p = blockIdx.z;  // the cluster spans blockIdx.y
    const size_t col0 = (size_t)blockIdx.x * W;
    const T *A = static_cast<const T *>(a.A) + p * a.stride_a;
    const T *x = static_cast<const T *>(a.x) + p * a.stride_x;
    const size_t j0 = min(seg * a.seg_len, a.N), j1 = min(j0 + a.seg_len, a.N);
    // Columns of this lane: CPL consecutive (VEC), or LPR apart.  A column past
    // the last is read as the last (VEC: M % CPL == 0, so whole vectors are in or
    // out) and not stored: loads under a condition would be waited for one by one.
    auto column = [&](int c) { return VEC ? lc * CPL + c : lc + c * LPR; };
    size_t off[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) off[c] = VEC ? min(col0 + lc * CPL, a.M - CPL) : min(col0 + column(c), a.M - 1);

    constexpr int NS = SETS ? SETS : 1;
    T acc[CPL], part[NS][CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
        acc[c] = T(0);
#pragma unroll
        for (int s = 0; s < NS; ++s) part[s][c] = T(0);
    }
    auto total = [&]() {  // the sets into the column's total
#pragma unroll
        for (int c = 0; c < CPL; ++c)
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                acc[c] += part[s][c];
                part[s][c] = T(0);
            }
    };
    constexpr int STEP = kWarps * RPW;  // rows per group of all warps
    size_t j = j0 + (size_t)w * RPW + lr;
    auto load = [&](const T *row, T (&v)[CPL]) {
        if constexpr (VEC) load_vec(row + off[0], v);
        else
#pragma unroll
            for (int c = 0; c < CPL; ++c) load_one(row + off[c], v[c]);
    };
    const T *row = A + j * a.lda;
    const size_t adv = (size_t)STEP * a.lda;
    for (; j + (size_t)(U - 1) * STEP < j1; j += (size_t)U * STEP, row += U * adv) {
        T v[U][CPL], xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            load(row + u * adv, v[u]);
            xv[u] = __ldg(x + j + (size_t)u * STEP);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < CPL; ++c) part[u % NS][c] = madd(v[u][c], xv[u], part[u % NS][c]);
        if (SETS == 0) total();
    }
    if (j < j1) {  // the last, partial group: rows past the segment are read as its last and add nothing
        T v[U][CPL], xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t r = min(j + (size_t)u * STEP, j1 - 1);
            load(A + r * a.lda, v[u]);
            xv[u] = __ldg(x + r);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = j + (size_t)u * STEP < j1;
#pragma unroll
            for (int c = 0; c < CPL; ++c) part[u % NS][c] = in ? madd(v[u][c], xv[u], part[u % NS][c]) : part[u % NS][c];
        }
    }
    total();
    // rows of a warp, then warps, then segments, each in a fixed order
#pragma unroll
    for (int off = LPR; off < 32; off <<= 1)
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
    if (lr == 0)
#pragma unroll
        for (int c = 0; c < CPL; ++c) red[w][column(c)] = acc[c];
    __syncthreads();
    if (threadIdx.x < W) {
        T t[kWarps];
#pragma unroll
        for (int ww = 0; ww < kWarps; ++ww) t[ww] = red[ww][threadIdx.x];
#pragma unroll
        for (int n = kWarps / 2; n > 0; n /= 2)
#pragma unroll
            for (int ww = 0; ww < n; ++ww) t[ww] = t[2 * ww] + t[2 * ww + 1];
        sums[threadIdx.x] = t[0];
    }
    const unsigned nseg = gridDim.y;
    if (nseg > 1) tc::cluster_sync();
    else __syncthreads();
    const size_t col = col0 + threadIdx.x;
    if (seg == 0 && threadIdx.x < W && col < a.M) {
        T t = sums[threadIdx.x];
        for (unsigned s = 1; s < nseg; ++s) {
            uint32_t addr;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(&sums[threadIdx.x])), "r"(s));
            t += ld_peer(addr, T(0));
        }
        T *y = static_cast<T *>(a.y) + p * a.stride_y + col;
        if (a.gemv) {
            const T beta = (T)a.beta;
            t = madd((T)a.alpha, t, beta == T(0) ? T(0) : beta * *y);
        }
        *y = t;
    }
    // no CTA leaves while the first may still read its sums
    if (nseg > 1) tc::cluster_sync();
}

}  // namespace gvc
}  // namespace gatlas
