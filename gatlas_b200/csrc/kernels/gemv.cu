// GEMV: y = A·x or y = alpha·A·x + beta·y, HBM streaming (buffer engine).
//
// Reference: KernelMatvecBuffer<SCALAR,VL>::print (KernelMatvecBuffer.hpp:180-325):
// one work item owns blockHeight rows and walks N/VL vectors of its rows and
// of b, accumulating with mad; transposeA reads A column-major
// (KernelMatvecBuffer.hpp:288-291).  Row-per-thread reads are uncoalesced for
// row-major A.
//
// B200 design (both layouts read every byte of A exactly once, 16-byte loads):
//  * trans_a == 0 (row-major): for long rows (at least 4 x 256 loads) a CTA
//    owns two rows at a time and its 256 threads stride across them in
//    16-byte vectors (single elements where rows are off the 16-byte grid),
//    reduced in a fixed order (warp butterfly, then the 8
//    warps in shared memory); otherwise a warp owns ROWS rows at a time, its
//    lanes striding across the row with UNROLL loads per row in flight and a
//    fixed butterfly shuffle reduction.  x is read through the L1-cached
//    read-only path.
//  * trans_a == 1 (column-major): one launch of clusters whose CTAs own the row
//    segments of a column block and add their sums over distributed shared
//    memory (gemv_cols.cuh) where the matrix has enough columns; otherwise a
//    CTA owns 32*VW adjacent columns (one
//    16-byte vector per lane) and one segment of the rows; its 8 warps take
//    interleaved rows, partial sums are combined across warps in a fixed order
//    in shared memory, and across the S row segments by the last CTA of each
//    column block (partials in a workspace, arrival counter per column block).
// Results are deterministic: the order depends only on (M, N) and the SM count.
// Measured (device time, before and after): 3001 x 7013 column-major 23.8 ->
// 17.2 us, row-major 45.6 -> 17.6; 1024 x 32767 207 -> 32; 1024^2 column-major
// 12.5 -> 4.3, row-major 4.5 -> 3.3; 32768 x 1024 column-major 36.5 -> 22.1.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "../common.cuh"
#include "../device_state.cuh"
#include "gemv_cols.cuh"

namespace gatlas {

template <typename T, int VW> struct VecT;
template <> struct VecT<float, 4> { using type = float4; };
template <> struct VecT<float, 1> { using type = float; };
template <> struct VecT<double, 2> { using type = double2; };
template <> struct VecT<double, 1> { using type = double; };

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// acc = fma chain over the vector's components in order.
__device__ __forceinline__ float dot_acc(float acc, float4 a, float4 x) {
    acc = fma_rn(a.x, x.x, acc);
    acc = fma_rn(a.y, x.y, acc);
    acc = fma_rn(a.z, x.z, acc);
    return fma_rn(a.w, x.w, acc);
}
__device__ __forceinline__ double dot_acc(double acc, double2 a, double2 x) {
    acc = fma_rn(a.x, x.x, acc);
    return fma_rn(a.y, x.y, acc);
}
__device__ __forceinline__ float dot_acc(float acc, float a, float x) { return fma_rn(a, x, acc); }
__device__ __forceinline__ double dot_acc(double acc, double a, double x) { return fma_rn(a, x, acc); }

template <typename T>
__device__ __forceinline__ T epilogue(int gemv, T alpha, T beta, T acc, const T *yold) {
    if (!gemv) return acc;
    const T bc = (beta == T(0)) ? T(0) : beta * (*yold);
    return fma_rn(alpha, acc, bc);
}

struct GemvArgs {
    const void *A;
    const void *x;
    void *y;
    size_t M, N, lda;
    size_t stride_a, stride_x, stride_y;
    double alpha, beta;
    int gemv;
};

constexpr int kGemvThreads = 256;
constexpr int kGemvWarps = kGemvThreads / 32;

// ---------------------------------------------------------------------------
// row-major A
// ---------------------------------------------------------------------------
// The last, partial group of a thread's strided vectors: all loads at once, as
// in a whole group, with vectors past the row read as its last one and left
// out of the sums (loading them one by one cost a memory latency each: rows of
// 32767 floats ran 207 us where rows of 32768 ran 26).
template <typename T, typename V, int ROWS, int UNROLL, int STRIDE>
__device__ __forceinline__ void row_tail(T (&acc)[ROWS], const V *const (&arow)[ROWS], const V *x, size_t c, size_t nvec) {
    V av[ROWS][UNROLL], xv[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
        const size_t i = min(c + (size_t)u * STRIDE, nvec - 1);
        xv[u] = __ldg(x + i);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) av[r][u] = __ldcs(arow[r] + i);
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
        const bool in = c + (size_t)u * STRIDE < nvec;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] = in ? dot_acc(acc[r], av[r][u], xv[u]) : acc[r];
    }
}

// One group of U strided vectors per row, all loads in flight together.
template <int U, int STRIDE, typename T, typename V, int ROWS>
__device__ __forceinline__ void row_group(T (&acc)[ROWS], const V *const (&arow)[ROWS], const V *x, size_t c) {
    V av[ROWS][U], xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) xv[u] = __ldg(x + c + u * STRIDE);
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int u = 0; u < U; ++u) av[r][u] = __ldcs(arow[r] + c + u * STRIDE);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] = dot_acc(acc[r], av[r][u], xv[u]);
}

// The rest of a row, up to U vectors a lane, as one group for the whole warp;
// only the last of them can be past the row, and is then read as the row's last
// vector and left out of the sums.  (Where some lanes held one more full group
// than others, the warp paid for both groups in turn, and a CTA waited three
// latencies for that warp instead of two: 8000 rows of 7200 floats ran 56 us, of
// 7168 39.)
template <int U, int STRIDE, typename T, typename V, int ROWS>
__device__ __forceinline__ void row_last(T (&acc)[ROWS], const V *const (&arow)[ROWS], const V *x, size_t c, int rem) {
    V av[ROWS][U], xv[U];
    const bool in = (U - 1) * STRIDE < rem;
    const int last = in ? (U - 1) * STRIDE : rem - 1;  // -1 and below: before c, inside the row all the same
#pragma unroll
    for (int u = 0; u < U; ++u) xv[u] = __ldg(x + c + (u < U - 1 ? u * STRIDE : last));
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int u = 0; u < U; ++u) av[r][u] = __ldcs(arow[r] + c + (u < U - 1 ? u * STRIDE : last));
#pragma unroll
    for (int u = 0; u < U - 1; ++u)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] = dot_acc(acc[r], av[r][u], xv[u]);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r] = in ? dot_acc(acc[r], av[r][U - 1], xv[U - 1]) : acc[r];
}

// Vectors c, c + STRIDE, ... of a row, four at a time; `first` is the warp's
// smallest c.
template <int STRIDE, typename T, typename V, int ROWS>
__device__ __forceinline__ void row_strided(T (&acc)[ROWS], const V *const (&arow)[ROWS], const V *x, size_t c,
                                            size_t first, size_t nvec) {
    for (; first + 31 + 3 * STRIDE < nvec; first += 4 * STRIDE, c += 4 * STRIDE) row_group<4, STRIDE>(acc, arow, x, c);
    if (first >= nvec) return;
    // the same small number twice: by warps the 64-bit form compiles to 48 registers,
    // by CTAs the 32-bit form (a difference of at most 4 * STRIDE, exact modulo 2^32)
    const int rem = STRIDE == 32 ? (int)((int64_t)nvec - (int64_t)c) : (int)nvec - (int)c;
    const int left = (int)(nvec - first);  // at most 4 * STRIDE
    if (left > 3 * STRIDE) row_last<4, STRIDE>(acc, arow, x, c, rem);
    else if (left > 2 * STRIDE) row_last<3, STRIDE>(acc, arow, x, c, rem);
    else if (left > STRIDE) row_last<2, STRIDE>(acc, arow, x, c, rem);
    else row_last<1, STRIDE>(acc, arow, x, c, rem);
}

// Vectors c, c + STRIDE, ... of a row, U at a time and the rest one by one.
// Written out, not through row_group: the compiler keeps more of a group's loads in
// flight this way (doubles off the 16-byte grid, 28440 x 4085: 176 us, 219
// through row_group), and a rest of one vector a lane costs less than row_last's
// clamped one (30000 x 4400 floats 86 us and 91).
template <int U, int STRIDE, typename T, typename V, int ROWS>
__device__ __forceinline__ void row_serial(T (&acc)[ROWS], const V *const (&arow)[ROWS], const V *x, size_t c, size_t nvec) {
    for (; c + (U - 1) * STRIDE < nvec; c += U * STRIDE) {
        V av[ROWS][U], xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) xv[u] = __ldg(x + c + u * STRIDE);
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u) av[r][u] = __ldcs(arow[r] + c + u * STRIDE);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] = dot_acc(acc[r], av[r][u], xv[u]);
    }
    for (; c < nvec; c += STRIDE) {
        const V xv = __ldg(x + c);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] = dot_acc(acc[r], __ldcs(arow[r] + c), xv);
    }
}

// FEW: few warps per SM, so the tail of a row loads at once (row_tail); with
// many its extra loads cost more (32768 x 1023: 29 us, 33 with row_tail; 1024^2
// the other way round).  Doubles are bound to 48 registers, five CTAs per SM.
template <typename T, int VW, int ROWS, int UNROLL, bool FEW>
__global__ void __launch_bounds__(kGemvThreads, VW == 2 ? 5 : 0)
    gemv_rows_kernel(GemvArgs a) {
    using V = typename VecT<T, VW>::type;
    const int lane = threadIdx.x & 31;
    const size_t warp = (size_t)blockIdx.x * kGemvWarps + (threadIdx.x >> 5);
    const size_t nwarps = (size_t)gridDim.x * kGemvWarps;
    const size_t p = blockIdx.y;
    const T *A = static_cast<const T *>(a.A) + p * a.stride_a;
    const V *x = reinterpret_cast<const V *>(static_cast<const T *>(a.x) + p * a.stride_x);
    T *y = static_cast<T *>(a.y) + p * a.stride_y;
    const size_t nvec = a.N / VW;
    const T alpha = (T)a.alpha, beta = (T)a.beta;

    for (size_t row0 = warp * ROWS; row0 < a.M; row0 += nwarps * ROWS) {
        T acc[ROWS];
        const V *arow[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            acc[r] = T(0);
            const size_t row = (row0 + r < a.M) ? row0 + r : a.M - 1;  // clamp; result discarded
            arow[r] = reinterpret_cast<const V *>(A + row * a.lda);
        }
        if constexpr (FEW) {
            size_t c = lane;
            for (; c + (UNROLL - 1) * 32 < nvec; c += UNROLL * 32) row_group<UNROLL, 32>(acc, arow, x, c);
            if (c < nvec) row_tail<T, V, ROWS, UNROLL, 32>(acc, arow, x, c, nvec);
        } else if constexpr (VW > 1) {
            static_assert(UNROLL == 4, "row_strided");
            row_strided<32>(acc, arow, x, lane, 0, nvec);
        } else {  // (row_strided: 32768 x 1023 floats 29 -> 41 us)
            row_serial<UNROLL, 32>(acc, arow, x, lane, nvec);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], off);
        }
        if (lane < ROWS) {
            T v = acc[0];
#pragma unroll
            for (int r = 1; r < ROWS; ++r)
                if (lane == r) v = acc[r];
            const size_t row = row0 + lane;
            if (row < a.M) y[row] = epilogue<T>(a.gemv, alpha, beta, v, y + row);
        }
    }
}

// Long rows: a CTA owns RB rows at a time and all 256 threads stride across
// each of them in 16-byte vectors (UNROLL per row in flight, x reused from
// registers across the RB rows); the per-thread chains are combined by a
// fixed butterfly per warp and a fixed-order sum over the 8 warps in shared
// memory.  The units are 8 times smaller than a warp's rows, so a 16384^2
// product is thousands of CTAs and the last partial wave costs little.
// SERIAL: the rest of a row one vector at a time (row_serial), else as one group
// (row_strided).  Both compile to 48 registers with 16-byte vectors, which is five
// CTAs per SM, without a bound that says so (at 56 16384^2 floats took 170 us, 166
// at 48); bounds on the float kernels spilled.
template <typename T, int VW, int RB, int UNROLL, bool SERIAL>
__global__ void __launch_bounds__(kGemvThreads)
    gemv_rowblock_kernel(GemvArgs a) {
    using V = typename VecT<T, VW>::type;
    __shared__ T red[RB][kGemvWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t p = blockIdx.y;
    const T *A = static_cast<const T *>(a.A) + p * a.stride_a;
    const V *x = reinterpret_cast<const V *>(static_cast<const T *>(a.x) + p * a.stride_x);
    T *y = static_cast<T *>(a.y) + p * a.stride_y;
    const size_t nvec = a.N / VW;
    const T alpha = (T)a.alpha, beta = (T)a.beta;
    const size_t nblocks = (a.M + RB - 1) / RB;
    for (size_t rb = blockIdx.x; rb < nblocks; rb += gridDim.x) {
        const size_t row0 = rb * RB;
        T acc[RB];
        const V *arow[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            acc[r] = T(0);
            const size_t row = (row0 + r < a.M) ? row0 + r : a.M - 1;  // clamp; result discarded
            arow[r] = reinterpret_cast<const V *>(A + row * a.lda);
        }
        if constexpr (VW == 1) {
            size_t c = threadIdx.x;
            for (; c + (UNROLL - 1) * kGemvThreads < nvec; c += UNROLL * kGemvThreads)
                row_group<UNROLL, kGemvThreads>(acc, arow, x, c);
            if (c < nvec) row_tail<T, V, RB, UNROLL, kGemvThreads>(acc, arow, x, c, nvec);
        } else if constexpr (SERIAL) {
            row_serial<UNROLL, kGemvThreads>(acc, arow, x, threadIdx.x, nvec);
        } else {
            static_assert(UNROLL == 4, "row_strided");
            row_strided<kGemvThreads>(acc, arow, x, threadIdx.x, w * 32, nvec);
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], off);
        }
        if (lane == 0)
#pragma unroll
            for (int r = 0; r < RB; ++r) red[r][w] = acc[r];
        __syncthreads();
        if (threadIdx.x < RB) {
            const int r = threadIdx.x;
            T v = red[r][0];
#pragma unroll
            for (int ww = 1; ww < kGemvWarps; ++ww) v += red[r][ww];
            const size_t row = row0 + r;
            if (row < a.M) y[row] = epilogue<T>(a.gemv, alpha, beta, v, y + row);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// column-major A
// ---------------------------------------------------------------------------
template <typename T, int VW, int UNROLL>
__global__ void __launch_bounds__(kGemvThreads)
    gemv_cols_kernel(GemvArgs a, int nseg, size_t seg_len, T *partial, unsigned *counters) {
    using V = typename VecT<T, VW>::type;
    __shared__ __align__(16) T red[kGemvWarps][32 * VW];
    __shared__ unsigned ticket;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const size_t cb = blockIdx.x, s = blockIdx.y, p = blockIdx.z;
    const size_t ncb = gridDim.x;
    const size_t col0 = cb * 32 * VW + (size_t)lane * VW;
    const bool active = col0 < a.M;  // M % VW == 0 is guaranteed when VW > 1
    const T *A = static_cast<const T *>(a.A) + p * a.stride_a;
    const T *x = static_cast<const T *>(a.x) + p * a.stride_x;
    T *y = static_cast<T *>(a.y) + p * a.stride_y;
    const size_t j0 = s * seg_len;
    const size_t j1 = (j0 + seg_len < a.N) ? j0 + seg_len : a.N;

    T acc[VW];
#pragma unroll
    for (int v = 0; v < VW; ++v) acc[v] = T(0);

    if (active) {
        size_t j = j0 + w;
        for (; j + (size_t)(UNROLL - 1) * kGemvWarps < j1; j += (size_t)UNROLL * kGemvWarps) {
            V av[UNROLL];
            T xv[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const size_t jj = j + (size_t)u * kGemvWarps;
                av[u] = __ldcs(reinterpret_cast<const V *>(A + jj * a.lda + col0));
                xv[u] = __ldg(x + jj);
            }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const T *e = reinterpret_cast<const T *>(&av[u]);
#pragma unroll
                for (int v = 0; v < VW; ++v) acc[v] = fma_rn(e[v], xv[u], acc[v]);
            }
        }
        for (; j < j1; j += kGemvWarps) {
            const V av = __ldcs(reinterpret_cast<const V *>(A + j * a.lda + col0));
            const T xv = __ldg(x + j);
            const T *e = reinterpret_cast<const T *>(&av);
#pragma unroll
            for (int v = 0; v < VW; ++v) acc[v] = fma_rn(e[v], xv, acc[v]);
        }
    }
#pragma unroll
    for (int v = 0; v < VW; ++v) red[w][lane * VW + v] = acc[v];
    __syncthreads();
    if (w != 0) return;

    T tot[VW];
#pragma unroll
    for (int v = 0; v < VW; ++v) {
        T t = red[0][lane * VW + v];
#pragma unroll
        for (int ww = 1; ww < kGemvWarps; ++ww) t += red[ww][lane * VW + v];
        tot[v] = t;
    }
    const T alpha = (T)a.alpha, beta = (T)a.beta;
    if (nseg == 1) {
        if (active)
#pragma unroll
            for (int v = 0; v < VW; ++v) y[col0 + v] = epilogue<T>(a.gemv, alpha, beta, tot[v], y + col0 + v);
        return;
    }
    // publish this segment's partial, then the last CTA of the column block sums
    T *part = partial + (p * nseg + s) * a.M;
    if (active)
#pragma unroll
        for (int v = 0; v < VW; ++v) part[col0 + v] = tot[v];
    __threadfence();
    __syncwarp();
    if (lane == 0) ticket = atomicAdd(counters + p * ncb + cb, 1u);
    __syncwarp();
    if (ticket != (unsigned)(nseg - 1)) return;
    __threadfence();
    if (!active) return;
#pragma unroll
    for (int v = 0; v < VW; ++v) {
        T t = T(0);
        for (int ss = 0; ss < nseg; ++ss) {
            const T pv = __ldcg(partial + (p * nseg + ss) * a.M + col0 + v);
            t = (ss == 0) ? pv : t + pv;
        }
        y[col0 + v] = epilogue<T>(a.gemv, alpha, beta, t, y + col0 + v);
    }
}

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
int matvec_image_f32(const gatlas_matvec_desc *d, const float *A, const float *x, float *y, void *ws,
                     size_t ws_bytes, cudaStream_t stream);
int matvec_image_f64(const gatlas_matvec_desc *d, const double *A, const double *x, double *y, void *ws,
                     size_t ws_bytes, cudaStream_t stream);
size_t matvec_image_ws_bytes(const gatlas_matvec_desc *d, size_t elem_bytes);

template <typename T>
static int matvec_image_dispatch(const gatlas_matvec_desc *d, const T *A, const T *x, T *y, void *ws,
                                 size_t ws_bytes, cudaStream_t stream) {
    if constexpr (sizeof(T) == 4) return matvec_image_f32(d, A, x, y, ws, ws_bytes, stream);
    else return matvec_image_f64(d, A, x, y, ws, ws_bytes, stream);
}

struct ColsPlan {
    int vw;
    size_t ncb, nseg, seg_len, part_bytes, counter_bytes;
};

template <typename T>
static ColsPlan cols_plan(const gatlas_matvec_desc *d, bool vec_ok) {
    ColsPlan pl{};
    const size_t batch = d->batch ? d->batch : 1;
    pl.vw = vec_ok ? (int)(16 / sizeof(T)) : 1;
    pl.ncb = (d->m + 32 * pl.vw - 1) / (32 * pl.vw);
    const size_t target = (size_t)sm_count() * 4;
    size_t per_batch = (target + batch - 1) / batch;
    size_t nseg = (per_batch + pl.ncb - 1) / pl.ncb;
    const size_t max_seg = (d->n + 31) / 32;
    if (nseg > max_seg) nseg = max_seg;
    if (nseg < 1) nseg = 1;
    if (nseg > 4096) nseg = 4096;
    if (d->n == 0) {
        pl.seg_len = 0;
        pl.nseg = 1;
    } else {
        pl.seg_len = (d->n + nseg - 1) / nseg;
        pl.nseg = (d->n + pl.seg_len - 1) / pl.seg_len;
    }
    if (pl.nseg > 1) {
        pl.part_bytes = (batch * pl.nseg * d->m * sizeof(T) + 255) & ~(size_t)255;
        pl.counter_bytes = (batch * pl.ncb * sizeof(unsigned) + 255) & ~(size_t)255;
    }
    return pl;
}

template <typename T>
static bool gemv_vec_ok(const gatlas_matvec_desc *d, const T *A, const T *x) {
    const size_t vw = 16 / sizeof(T);
    const size_t lda = d->lda ? d->lda : (d->trans_a ? d->m : d->n);
    const size_t inner = d->trans_a ? d->m : d->n;
    const size_t batch = d->batch ? d->batch : 1;
    bool ok = aligned16(A) && (lda % vw == 0) && (inner % vw == 0);
    if (!d->trans_a) ok = ok && aligned16(x);
    if (batch > 1) {
        const size_t sa = d->stride_a ? d->stride_a : lda * (d->trans_a ? d->n : d->m);
        const size_t sx = d->stride_x ? d->stride_x : d->n;
        ok = ok && (sa % vw == 0) && (d->trans_a || sx % vw == 0);
    }
    return ok;
}

// Column-major products whose segments fit one cluster (gemv_cols.cuh).
constexpr int kMaxSegments = 8;  // CTAs of a portable cluster
struct ClusterKernel {
    const void *fn;
    size_t width;                                     // columns per block
    bool even;                                        // segments dealt evenly to SMs (see cluster_plan)
    std::atomic<int> resident[64][kMaxSegments + 1];  // per device and cluster size, 0: not asked yet
};
struct ClusterPlan {
    const ClusterKernel *kernel;
    int nseg;  // 0: the general kernel, with partial sums in a workspace
};

static cudaLaunchConfig_t cluster_config(dim3 grid, int nseg, cudaLaunchAttribute *attr, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(gvc::kThreads, 1, 1);
    cfg.stream = stream;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = 1;
    attr->val.clusterDim.y = (unsigned)nseg;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Clusters of nseg CTAs that the current device (dev) holds at once.  Fewer than its
// CTAs over nseg, since a cluster needs its CTAs in one place: three CTAs per SM
// make 222 clusters of 2, but 104 of 4 and 48 of 8.  With one cluster more a second
// wave nearly doubles the time (3396 x 27644 doubles: 111 us at 0.92 of what
// fits, 149 at 1.10).
static size_t clusters_resident(ClusterKernel &k, int dev, int nseg) {
    std::atomic<int> &known = k.resident[dev & 63][nseg];
    int n = known.load(std::memory_order_relaxed);
    if (n == 0) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = cluster_config(dim3(1, (unsigned)nseg, 1), nseg, &attr, nullptr);
        if (cudaOccupancyMaxActiveClusters(&n, k.fn, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            n = std::max(1, sm_count() * 2 / nseg);
        }
        known.store(n, std::memory_order_relaxed);
    }
    return (size_t)n;
}

// The kernel by columns (times instances), then as many segments as fit at once,
// of 256 rows at least (2602 x 517 floats 6.2 us, 7.2 in 8 segments), 512 of up to 64
// floats where the blocks alone fill the SMs (13676 x 992 8.2 us, 10.2 in two).
template <typename T>
static ClusterPlan cluster_plan(const gatlas_matvec_desc *d, bool vec_ok) {
    constexpr int V = 16 / (int)sizeof(T);
    const ClusterPlan general{nullptr, 0};
    const size_t batch = d->batch ? d->batch : 1, sms = (size_t)sm_count();
    const auto blocks_of = [&](size_t width) { return (d->m + width - 1) / width * batch; };
    if (d->n == 0 || blocks_of(32) * 8 < sms) return general;  // too few blocks for clusters of 8
    int dev = 0;
    cudaGetDevice(&dev);
    const auto segments = [&](ClusterKernel &k) {
        const size_t rows = sizeof(T) == 4 && k.width <= 64 && blocks_of(k.width) >= sms ? 512 : 256;
        int s = kMaxSegments;
        while (s > 1 && ((size_t)s * rows > d->n || blocks_of(k.width) > clusters_resident(k, dev, s))) --s;
        return s;
    };
    // blocks over what fits at once, and that over whole waves
    const auto fill = [&](ClusterKernel &k, int s) { return (double)blocks_of(k.width) / (double)clusters_resident(k, dev, s); };
    const auto wave_share = [](double f) { return f / std::ceil(f); };
    ClusterKernel *k;
    if constexpr (sizeof(T) == 4) {
        static ClusterKernel vec[] = {{(const void *)gvc::gemv_cols_cluster_kernel<T, true, 8, V, 16, 0, 0>, 32, false, {}},
                                      {(const void *)gvc::gemv_cols_cluster_kernel<T, true, 16, V, 16, 0, 0>, 64, false, {}},
                                      {(const void *)gvc::gemv_cols_cluster_kernel<T, true, 32, V, 8, 0, 0>, 128, false, {}}};
        static ClusterKernel one[] = {{(const void *)gvc::gemv_cols_cluster_kernel<T, false, 16, 2, 16, 0, 0>, 32, true, {}},
                                      {(const void *)gvc::gemv_cols_cluster_kernel<T, false, 32, 2, 16, 0, 0>, 64, false, {}},
                                      {(const void *)gvc::gemv_cols_cluster_kernel<T, false, 16, 4, 8, 1, 0>, 64, false, {}},
                                      {(const void *)gemv_cols_kernel<T, 1, 4>, 32, false, {}}};
        if (vec_ok) {
            // 32 columns until clusters of 8 on 64 columns fill half the GPU (868 x
            // 10563 9.1 us against 10.2, 1116 x 56216 49 and 53; 1524 x 1905 8.3 and
            // 6.3), then 64 until clusters of two just fit (12000 x 10000 72 us, 128
            // columns 74; 13604 x 14780 123 and 118; 30000 x 4000 90 and 74), or while
            // they fit where columns are short (17236 x 452 6.2 and 8.2).  Long columns
            // again where single CTAs of 128 are under 2/3 of what fits or over it
            // (40000 x 6000 147 and 157, 100000 x 2000 120 and 132; 60000 x 500 25 and
            // 22); just over it the general kernel (80000 x 1000 48 us, 64 columns 52).
            const bool brief = d->n < 1024;
            const double f128 = fill(vec[2], 1);
            if (f128 > 1 && f128 <= 1.25) return general;
            if (blocks_of(64) * 2 < clusters_resident(vec[1], dev, 8)) k = &vec[0];
            else if (fill(vec[1], 2) <= 0.9 || (brief && fill(vec[1], 1) <= 1)) k = &vec[1];
            else k = &vec[brief || fill(vec[2], 2) <= 1 || (f128 * 3 > 2 && f128 <= 1) ? 2 : 1];
        } else if (blocks_of(32) * 2 <= sms) {
            // off the 16-byte grid: 32 columns up to half a block per SM (1001 x 30001
            // 29 us, 64 columns 45; 2203 x 30011 52 and 54; 3301 x 20003 52 and 50)
            k = &one[0];
        } else {
            // 64 columns: 16 rows in flight, or 8 where columns are short (3001 x 7013 17.3
            // us and 16.5, 9001 x 3001 21.4 and 20.6; 5001 x 14003 50 and 52) or more CTAs
            // then fill the GPU better (15001 x 9001 110 and 95)
            const int s1 = segments(one[1]), s2 = segments(one[2]);
            k = &one[d->n < 8192 || fill(one[2], s2) > fill(one[1], s1) + 0.1 ? 2 : 1];
            // from about 20800 columns the general kernel's many small CTAs are faster
            // (22003 x 3001 46 us and 49) unless their last wave is nearly empty (30001 x
            // 4001 113 and 83)
            if (blocks_of(64) * 10 > sms * 22) {
                k = &one[2];
                if (wave_share(fill(one[3], 1)) * 1.1 >= wave_share(fill(one[2], 1))) return general;
            }
        }
    } else {
        static ClusterKernel vec[] = {{(const void *)gvc::gemv_cols_cluster_kernel<T, true, 16, V, 8, 2, 5>, 32, false, {}},
                                      {(const void *)gvc::gemv_cols_cluster_kernel<T, true, 32, V, 8, 2, 5>, 64, false, {}},
                                      {(const void *)gvc::gemv_cols_cluster_kernel<T, true, 16, V, 8, 2, 6>, 32, false, {}}};
        // off the 16-byte grid the general kernel is faster (2479 x 5702: 26 us against 33)
        if (!vec_ok) return general;
        // 32 columns until clusters of 8 on 64 fill three quarters of the GPU (3872 x
        // 16820 79 us, 64 columns 82; 6732 x 5348 49 and 47), while they fit where
        // columns are short, and again where blocks of 64 no longer fit (44728 x 4940 255
        // and 251; 59288 x 2516 179 and 196) unless the last wave is nearly empty (50002
        // x 5002 331, general kernel 293; 56388 x 3720, 0.4 full, 252 and 269)
        const double f32 = fill(vec[0], 1), f64 = fill(vec[1], 1);
        if (f64 > 1 && f32 - std::floor(f32) < 0.33) return general;
        if (f32 > 1 && fill(vec[2], 1) <= 1) k = &vec[2];
        else k = &vec[blocks_of(64) * 4 > clusters_resident(vec[1], dev, 8) * 3 && f64 <= 1 && (d->n >= 512 || f32 > 1) ? 1 : 0];
    }
    const size_t blocks = blocks_of(k->width);
    if (blocks * 8 < sms || blocks / batch > 0x7fffffffu) return general;
    int nseg = segments(*k);
    // The narrow kernel off the 16-byte grid is bound by the SM with the most rows:
    // whole CTAs per SM (3 % fewer SMs, since clusters do not pack them all) over the
    // segment count (1617 x 13049, 51 blocks: 18.6 us with 5 segments, 20.6 with 7;
    // 1411 x 40003, 45: 45 with 6, 49 with 8).
    if (k->even) {
        const size_t even_sms = sms * 97 / 100;
        const auto load = [&](int s) { return (double)((blocks * s + even_sms - 1) / even_sms) / s; };
        for (int s = nseg - 1; s >= 1; --s)
            if (load(s) < load(nseg)) nseg = s;
    }
    // few columns and long rows of doubles: the general kernel cuts the rows finer,
    // as fast (1450 x 31575: 66 us both, 1392 x 10148 25 and 27) and with shorter sums
    if (sizeof(T) == 8 && nseg == 8 && blocks * 8 < 3 * sms && d->n >= 9216) return general;
    return {k, nseg};
}

static int launch_cluster(const GemvArgs &g, const ClusterPlan &cp, size_t batch, cudaStream_t stream) {
    gvc::Args a;
    a.A = g.A, a.x = g.x, a.y = g.y;
    a.M = g.M, a.N = g.N, a.lda = g.lda;
    a.stride_a = g.stride_a, a.stride_x = g.stride_x, a.stride_y = g.stride_y;
    a.alpha = g.alpha, a.beta = g.beta, a.gemv = g.gemv;
    a.seg_len = (g.N + cp.nseg - 1) / cp.nseg;
    const size_t width = cp.kernel->width;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config(
        dim3((unsigned)((g.M + width - 1) / width), (unsigned)cp.nseg, (unsigned)batch), cp.nseg, &attr, stream);
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, cp.kernel->fn, args);
    if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "gemv_cols_cluster_kernel: %s", cudaGetErrorString(e));
    return check_launch("gemv_cols_cluster_kernel");
}

bool matvec_buffer_scratchless(const gatlas_matvec_desc *d, size_t elem_bytes) {
    if (!d->trans_a) return true;
    return (elem_bytes == 4 ? cluster_plan<float>(d, true) : cluster_plan<double>(d, true)).nseg > 0;
}

template <typename T>
static size_t matvec_ws(const gatlas_matvec_desc *d, const void *A, const void *x) {
    if (!d || !d->trans_a) return 0;
    if (d->engine == GATLAS_ENGINE_IMAGE) return matvec_image_ws_bytes(d, sizeof(T));
    const ColsPlan pl = cols_plan<T>(d, gemv_vec_ok<T>(d, (const T *)A, (const T *)x));
    return pl.part_bytes + pl.counter_bytes;
}

template <typename T>
static int matvec_launch(const gatlas_matvec_desc *d, const T *A, const T *x, T *y, void *ws,
                         size_t ws_bytes, cudaStream_t stream) {
    if (!d) return set_error(GATLAS_ERR_INVALID, "matvec: null descriptor");
    if (d->engine == GATLAS_ENGINE_IMAGE) return matvec_image_dispatch<T>(d, A, x, y, ws, ws_bytes, stream);
    if (d->engine != GATLAS_ENGINE_BUFFER)
        return set_error(GATLAS_ERR_INVALID, "matvec: engine %d is not buffer/image", d->engine);
    if (d->m == 0) return GATLAS_OK;
    if (!A || !x || !y) return set_error(GATLAS_ERR_INVALID, "matvec: null pointer");
    const size_t batch = d->batch ? d->batch : 1;
    if (batch > 65535) return set_error(GATLAS_ERR_INVALID, "matvec: batch %zu > 65535", batch);
    const size_t lda = d->lda ? d->lda : (d->trans_a ? d->m : d->n);
    if ((!d->trans_a && lda < d->n) || (d->trans_a && lda < d->m))
        return set_error(GATLAS_ERR_INVALID, "matvec: lda %zu too small", lda);

    GemvArgs a;
    a.A = A;
    a.x = x;
    a.y = y;
    a.M = d->m;
    a.N = d->n;
    a.lda = lda;
    a.stride_a = d->stride_a ? d->stride_a : lda * (d->trans_a ? d->n : d->m);
    a.stride_x = d->stride_x ? d->stride_x : d->n;
    a.stride_y = d->stride_y ? d->stride_y : d->m;
    a.alpha = d->alpha;
    a.beta = d->beta;
    a.gemv = d->gemv;

    const bool vec_ok = gemv_vec_ok<T>(d, A, x);
    const int sms = sm_count();
    if (!d->trans_a) {
        constexpr int VWV = 16 / sizeof(T);
        const size_t per_row = vec_ok ? d->n / VWV : d->n;  // loads per row
        // long rows take a CTA per RB rows: 1024 vectors, or as many single elements
        // unless there are rows enough for a warp each.  How many that takes grows with
        // the row (floats 7500 x 2049 10 us with warps, 14 with CTAs, 9000 x 3001 25 and
        // 29, 9000 x 3502 31 and 30; doubles 7001 x 1201 12 and 14, 6000 x 2343 31 and 27,
        // 9000 x 2343 36 and 39, 9000 x 3503 51 and 45; 27908 x 1287 58 and 62)
        constexpr size_t kT = kGemvThreads;
        const size_t rows_all = d->m * batch;
        const size_t warps_from = (size_t)sms * (sizeof(T) == 4 ? (per_row < 8 * kT ? 32 : per_row < 13 * kT ? 27 : 64)
                                                                : (per_row < 8 * kT ? 32 : per_row < 11 * kT ? 48 : 64));
        // (12000 x 4501 43 and 49, 16000 x 4501 72 and 64)
        const bool many = rows_all >= warps_from &&
                          (per_row < 16 * kT || (sizeof(T) == 4 && per_row < 20 * kT && rows_all < (size_t)sms * 96));
        if (per_row >= (size_t)4 * kGemvThreads && (vec_ok || !many)) {
            // (single elements: twice as many in flight where the row holds them)
            constexpr int RB = 2;
            const size_t nblocks = (d->m + RB - 1) / RB;
            const size_t cap = (size_t)sms * 64 / (batch < 8 ? batch : 8);
            dim3 g((unsigned)(nblocks < cap ? nblocks : cap), (unsigned)batch);
            // row_serial where rows end soon after the first group (doubles: first two), by
            // not much more than one vector a thread (15000 x 4100 floats 43.5 us, 46 through
            // row_strided, 5264 x 5244 21 and 22; but 25164 x 8924 140 and 132, 10000 columns
            // 81 and 76, 7200 58 and 41), doubles in few rows also after more groups (1500 x
            // 8200 21 and 22), and long rows of them with any rest (568 x 26424 29 and 32,
            // 1126 x 46736 72 and 71)
            const size_t rest = per_row % (4 * kT);
            const bool few_f64 = sizeof(T) == 8 && rows_all <= (size_t)sms * 12;
            const bool serial = (rest > 0 && rest * 4 < 5 * kT && (per_row < (sizeof(T) == 8 ? 12 : 8) * kT || few_f64)) ||
                                (few_f64 && rows_all <= (size_t)sms * 7 && per_row >= 32 * kT);
            if (vec_ok && serial) gemv_rowblock_kernel<T, VWV, RB, 4, true><<<g, kGemvThreads, 0, stream>>>(a);
            else if (vec_ok) gemv_rowblock_kernel<T, VWV, RB, 4, false><<<g, kGemvThreads, 0, stream>>>(a);
            else if (per_row >= (size_t)8 * kGemvThreads)
                gemv_rowblock_kernel<T, 1, RB, 8, false><<<g, kGemvThreads, 0, stream>>>(a);
            else gemv_rowblock_kernel<T, 1, RB, 4, false><<<g, kGemvThreads, 0, stream>>>(a);
            return check_launch("gemv_rowblock_kernel");
        }
        // shorter rows: a warp per two rows, or per row (and twice the loads of
        // it in flight) while that leaves SMs with few warps: up to about one wave
        // of it, five CTAs per SM, and again where two rows a warp just begin a
        // second wave (N = 3500: M = 6200 13 us and 17 with two rows, 7400 22 and
        // 19, 11000 28 and 25, 13000 32 and 36, 18000 51 and 43)
        const size_t wave = 5 * kGemvWarps * (size_t)sms;
        const bool few = rows_all < (size_t)sms * 4 * kGemvWarps ||
                         (vec_ok && (rows_all * 20 <= wave * (sizeof(T) == 8 ? 21 : 23) ||
                                     (rows_all > 2 * wave && rows_all * 10 <= wave * 24)));
        const int rows = few ? 1 : 2;
        const size_t warps_needed = (d->m + rows - 1) / rows;
        size_t grid = (warps_needed + kGemvWarps - 1) / kGemvWarps;
        const size_t cap = (size_t)sms * 8 / (batch < 8 ? batch : 8);
        if (grid > cap) grid = cap ? cap : 1;
        dim3 g((unsigned)grid, (unsigned)batch);
        if (vec_ok) {
            if (few) gemv_rows_kernel<T, VWV, 1, 8, true><<<g, kGemvThreads, 0, stream>>>(a);
            else gemv_rows_kernel<T, VWV, 2, 4, false><<<g, kGemvThreads, 0, stream>>>(a);
        } else {
            if (few) gemv_rows_kernel<T, 1, 1, 16, true><<<g, kGemvThreads, 0, stream>>>(a);
            else gemv_rows_kernel<T, 1, 2, 4, false><<<g, kGemvThreads, 0, stream>>>(a);
        }
        return check_launch("gemv_rows_kernel");
    }

    const ColsPlan pl = cols_plan<T>(d, vec_ok);
    T *partial = nullptr;
    unsigned *counters = nullptr;
    if (pl.nseg > 1) {
        const size_t need = pl.part_bytes + pl.counter_bytes;
        if (ws && ws_bytes < need)
            return set_error(GATLAS_ERR_INVALID, "matvec: workspace %zu < %zu bytes", ws_bytes, need);
        if (ws && !aligned_to(ws, 256)) return set_error(GATLAS_ERR_INVALID, "matvec: workspace must be 256-byte aligned");
    }
    if (const ClusterPlan cp = cluster_plan<T>(d, vec_ok); cp.nseg) return launch_cluster(a, cp, batch, stream);
    if (pl.nseg > 1) {
        const size_t need = pl.part_bytes + pl.counter_bytes;
        if (!ws) {
            ws = device_scratch(need);
            if (!ws) return set_error(GATLAS_ERR_NOMEM, "matvec: scratch of %zu bytes", need);
        }
        partial = static_cast<T *>(ws);
        counters = reinterpret_cast<unsigned *>(static_cast<char *>(ws) + pl.part_bytes);
        cudaError_t e = cudaMemsetAsync(counters, 0, pl.counter_bytes, stream);
        if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "matvec: memset counters: %s", cudaGetErrorString(e));
    }
    dim3 g((unsigned)pl.ncb, (unsigned)pl.nseg, (unsigned)batch);
    if (pl.ncb > 0x7fffffffu || pl.nseg > 65535)
        return set_error(GATLAS_ERR_INVALID, "matvec: grid too large");
    if (pl.vw > 1) {
        constexpr int VW = 16 / sizeof(T);
        gemv_cols_kernel<T, VW, 4><<<g, kGemvThreads, 0, stream>>>(a, (int)pl.nseg, pl.seg_len, partial, counters);
    } else {
        gemv_cols_kernel<T, 1, 4><<<g, kGemvThreads, 0, stream>>>(a, (int)pl.nseg, pl.seg_len, partial, counters);
    }
    return check_launch("gemv_cols_kernel");
}

}  // namespace gatlas

extern "C" size_t gatlas_matvec_workspace_size(const gatlas_matvec_desc *d) {
    // The largest need over both element types and both load widths, so the
    // answer holds whichever path the launch picks.
    if (!d || !d->trans_a) return 0;
    size_t best = 0;
    for (int vec = 0; vec < 2; ++vec) {
        const gatlas::ColsPlan f = gatlas::cols_plan<float>(d, vec != 0);
        const gatlas::ColsPlan g = gatlas::cols_plan<double>(d, vec != 0);
        const size_t a = f.part_bytes + f.counter_bytes, b = g.part_bytes + g.counter_bytes;
        if (a > best) best = a;
        if (b > best) best = b;
    }
    const size_t img = std::max(gatlas::matvec_image_ws_bytes(d, 4), gatlas::matvec_image_ws_bytes(d, 8));
    return img > best ? img : best;
}

extern "C" int gatlas_matvec_f32(const gatlas_matvec_desc *d, const float *A, const float *x, float *y,
                                 void *workspace, size_t workspace_bytes, void *stream) {
    return gatlas::matvec_launch<float>(d, A, x, y, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int gatlas_matvec_f64(const gatlas_matvec_desc *d, const double *A, const double *x,
                                 double *y, void *workspace, size_t workspace_bytes, void *stream) {
    return gatlas::matvec_launch<double>(d, A, x, y, workspace, workspace_bytes, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Allocation-free GEMV entry point.
//
// For callers that cannot call cudaMalloc: code that runs inside a host
// framework which owns all device memory (or has reserved it for its own
// pool), and code on a latency-critical path that must not trigger the
// device-wide synchronisation cudaMalloc/cudaFree imply.  The column-major
// path needs scratch for per-segment partial sums and arrival counters; this
// entry point takes it from a fixed 1 MiB array in device memory that this
// file owns, instead of from a workspace or the library's allocation cache.
// ---------------------------------------------------------------------------
#include <mutex>

namespace gatlas {
namespace {

constexpr size_t kNoAllocScratchBytes = GATLAS_MATVEC_NOALLOC_SCRATCH_BYTES;

// One copy per GPU that loads this library, held until the process exits.
// Host code may not use this name as a device address: the device address is
// looked up once per device with cudaGetSymbolAddress.
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void *g_noalloc_ptr[kNoAllocMaxDevices] = {nullptr};

// Device address of g_noalloc_scratch for the current device (looked up on
// the first call on each device, with that device current).
int noalloc_scratch(void **out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "matvec_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return set_error(GATLAS_ERR_INVALID, "matvec_noalloc: device %d", dev);
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return set_error(GATLAS_ERR_CUDA, "matvec_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return GATLAS_OK;
}

}  // namespace
}  // namespace gatlas

extern "C" int gatlas_matvec_f32_noalloc(const gatlas_matvec_desc *d, const float *A, const float *x, float *y,
                                         void *stream) {
    using namespace gatlas;
    if (!d) return set_error(GATLAS_ERR_INVALID, "matvec_noalloc: null descriptor");
    const size_t need = matvec_ws<float>(d, A, x);
    if (need > kNoAllocScratchBytes)
        return set_error(GATLAS_ERR_INVALID,
                         "matvec_noalloc: this problem needs %zu bytes of scratch, more than the %zu-byte "
                         "static scratch of the allocation-free entry point; call gatlas_matvec_f32 with a "
                         "workspace instead",
                         need, kNoAllocScratchBytes);
    void *scratch = nullptr;
    const int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    return matvec_launch<float>(d, A, x, y, scratch, kNoAllocScratchBytes, (cudaStream_t)stream);
}
