// Launch of the FP32 asynchronous-copy GEMM (gemm_ffma.cuh): tile choice and grid.
#include <algorithm>
#include <atomic>

#include "gemm_engines.hpp"
#include "gemm_ffma.cuh"

namespace gatlas {

namespace {

// Tilings: tile, micro-tile, lanes along m, CTAs per SM asked for, whether a
// step's first fragments load a step ahead (it costs the registers the widest
// micro-tile needs).
struct Large {
    static constexpr int BM = 128, BN = 128, TM = 8, TN = 16, LM = 8, MINB = 2, STAGES = 3;
    static constexpr bool AHEAD = false;
};
struct Medium {
    static constexpr int BM = 128, BN = 64, TM = 8, TN = 8, LM = 4, MINB = 2, STAGES = 4;
    static constexpr bool AHEAD = true;
};
struct Small {
    static constexpr int BM = 64, BN = 64, TM = 8, TN = 4, LM = 4, MINB = 3, STAGES = 4;
    static constexpr bool AHEAD = true;
};
struct Tiny {
    static constexpr int BM = 32, BN = 32, TM = 4, TN = 4, LM = 4, MINB = 6, STAGES = 4;
    static constexpr bool AHEAD = true;
};

template <typename P, bool TA, bool TB>
int launch(ffma::Args a, int64_t batch, cudaStream_t stream) {
    // a turned B is needed a step earlier: one more stage at least
    constexpr int STAGES = TB && P::STAGES < 4 ? P::STAGES + 1 : P::STAGES;
    auto kern = ffma::gemm_ffma_kernel<P::BM, P::BN, P::TM, P::TN, P::LM, TA, TB, STAGES, P::MINB, P::AHEAD>;
    constexpr int smem = ffma::smem_bytes<P::BM, P::BN, TA, TB, STAGES>();
    static std::atomic<uint64_t> configured{0};  // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "gemm_ffma smem attribute: %s", cudaGetErrorString(e));
        configured.fetch_or(bit, std::memory_order_release);
    }
    a.tiles_m = (int)((a.M + P::BM - 1) / P::BM);
    a.tiles_n = (int)((a.N + P::BN - 1) / P::BN);
    const dim3 grid((unsigned)((int64_t)a.tiles_m * a.tiles_n), 1, (unsigned)batch);
    kern<<<grid, P::BM / P::TM * (P::BN / P::TN), smem, stream>>>(a);
    return check_launch("gemm_ffma_kernel");
}

template <typename P>
int launch_layout(const Geometry &g, const ffma::Args &a, cudaStream_t stream) {
    if (g.ta) return g.tb ? launch<P, true, true>(a, g.batch, stream) : launch<P, true, false>(a, g.batch, stream);
    return g.tb ? launch<P, false, true>(a, g.batch, stream) : launch<P, false, false>(a, g.batch, stream);
}

// Time of a tiling in elements of C per SM over its rate: `rate` is its
// TFLOP/s at 4096 x 4096 x 2048 (53, 51, 48 and 40), `fill[i]` the share of
// that which an SM with i + 1 of its CTAs reaches (from 1024^3: 108, 62, 64
// and 72 us; 512^3: 55, 32, 23 and 15; 256^3: 31, 19, 12 and 8; 64 x 3000 x
// 1024: 109, 62, 41 and 27), the last entry its full residency.
template <typename P>
double tiling_cost(const Geometry &g, double rate, const double *fill, int residency) {
    const int64_t tiles = ((g.M + P::BM - 1) / P::BM) * ((g.N + P::BN - 1) / P::BN) * g.batch;
    const int64_t per_sm = (tiles + sm_count() - 1) / sm_count();
    const int64_t whole = per_sm / residency * residency, rest = per_sm - whole;
    const double units = (double)whole + (rest ? (double)rest / fill[rest - 1] : 0.0);
    return units * (P::BM * P::BN) / rate;
}

}  // namespace

bool matmul_ffma_takes(const Geometry &g) {
    // grids of the smallest tile fit in x, and no more rows of C than the SIMT
    // default's grid takes (65535 tiles of 128 rows)
    return (g.M + 127) / 128 <= 65535 && ((g.M + 31) / 32) * ((g.N + 31) / 32) <= (1 << 27);
}

int matmul_ffma(const gatlas_matmul_desc *d, const Geometry &g, const float *A, const float *B, float *C,
                cudaStream_t stream) {
    ffma::Args a;
    a.A = A, a.B = B, a.C = C;
    a.M = g.M, a.N = g.N, a.K = g.K;
    a.lda = g.lda, a.ldb = g.ldb, a.ldc = g.ldc;
    a.stride_a = g.stride_a, a.stride_b = g.stride_b, a.stride_c = g.stride_c;
    a.alpha = (float)d->alpha, a.beta = (float)d->beta, a.gemm = d->gemm;
    a.vec_a = aligned16(A) && g.lda % 4 == 0 && (g.batch == 1 || g.stride_a % 4 == 0);
    a.vec_b = aligned16(B) && g.ldb % 4 == 0 && (g.batch == 1 || g.stride_b % 4 == 0);
    a.tiles_m = a.tiles_n = 0;
    static const double kLarge[] = {0.88, 1.0}, kMedium[] = {0.83, 1.0}, kSmall[] = {0.66, 0.85, 1.0},
                        kTiny[] = {0.37, 0.57, 0.72, 0.82, 0.92, 1.0};
    const double large = tiling_cost<Large>(g, 53, kLarge, 2), medium = tiling_cost<Medium>(g, 51, kMedium, 2);
    const double small = tiling_cost<Small>(g, 48, kSmall, 3), tiny = tiling_cost<Tiny>(g, 40, kTiny, 6);
    const double best = std::min(std::min(large, medium), std::min(small, tiny));
    if (best == large) return launch_layout<Large>(g, a, stream);
    if (best == medium) return launch_layout<Medium>(g, a, stream);
    if (best == small) return launch_layout<Small>(g, a, stream);
    return launch_layout<Tiny>(g, a, stream);
}

}  // namespace gatlas
