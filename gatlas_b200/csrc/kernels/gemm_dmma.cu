// Launch of the FP64 tensor-core GEMM (gemm_dmma.cuh): tile choice and grid.
#include <atomic>

#include "gemm_dmma.cuh"
#include "gemm_engines.hpp"

namespace gatlas {

namespace {

template <int BM, int BN, int WM, int WN, bool TA, bool TB>
int launch(dmma::Args a, int64_t batch, cudaStream_t stream) {
    auto kern = dmma::gemm_dmma_kernel<BM, BN, WM, WN, TA, TB>;
    constexpr int smem = dmma::smem_bytes<BM, BN, TA, TB>();
    static std::atomic<uint64_t> configured{0};  // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return set_error(GATLAS_ERR_CUDA, "gemm_dmma smem attribute: %s", cudaGetErrorString(e));
        configured.fetch_or(bit, std::memory_order_release);
    }
    a.tiles_m = (int)((a.M + BM - 1) / BM);
    a.tiles_n = (int)((a.N + BN - 1) / BN);
    const dim3 grid((unsigned)((int64_t)a.tiles_m * a.tiles_n), 1, (unsigned)batch);
    kern<<<grid, BM / WM * (BN / WN) * 32, smem, stream>>>(a);
    return check_launch("gemm_dmma_kernel");
}

template <int BM, int BN, int WM, int WN>
int launch_layout(const Geometry &g, const dmma::Args &a, cudaStream_t stream) {
    if (g.ta) return g.tb ? launch<BM, BN, WM, WN, true, true>(a, g.batch, stream)
                          : launch<BM, BN, WM, WN, true, false>(a, g.batch, stream);
    return g.tb ? launch<BM, BN, WM, WN, false, true>(a, g.batch, stream)
                : launch<BM, BN, WM, WN, false, false>(a, g.batch, stream);
}

// Time of a tiling in multiply-adds per SM over its rate.  The rates are the
// TFLOP/s of 4096 x 4096 x 2048 (64 x 64: 33.4, 64 x 32: 30.9, 32 x 32: 29.3;
// 128 x 128 with 256 threads ran 31.9 and lost everywhere); an SM that holds
// one or two CTAs hides less latency (512^3: 29.2, 19.0 and 17.0 us for the
// three; 1000 x 600 x 2000: 150, 130 and 117; 2047^2 x 511: 142, 153 and 164).
double tiling_cost(int64_t tiles, double area, double rate) {
    const int64_t per_sm = (tiles + sm_count() - 1) / sm_count();
    return (double)per_sm * area / rate * (per_sm == 1 ? 1.6 : per_sm == 2 ? 1.3 : 1.0);
}

}  // namespace

bool matmul_dmma_takes(const Geometry &g) {
    // grids of the smallest tile fit in x, and no more rows of C than the SIMT
    // kernel's grid takes (65535 tiles of 64 rows)
    return (g.M + 63) / 64 <= 65535 && ((g.M + 31) / 32) * ((g.N + 31) / 32) <= (1 << 27);
}

int matmul_dmma(const gatlas_matmul_desc *d, const Geometry &g, const double *A, const double *B, double *C,
                cudaStream_t stream) {
    dmma::Args a;
    a.A = A, a.B = B, a.C = C;
    a.M = g.M, a.N = g.N, a.K = g.K;
    a.lda = g.lda, a.ldb = g.ldb, a.ldc = g.ldc;
    a.stride_a = g.stride_a, a.stride_b = g.stride_b, a.stride_c = g.stride_c;
    a.alpha = d->alpha, a.beta = d->beta, a.gemm = d->gemm;
    a.vec_a = aligned16(A) && g.lda % 2 == 0 && (g.batch == 1 || g.stride_a % 2 == 0);
    a.vec_b = aligned16(B) && g.ldb % 2 == 0 && (g.batch == 1 || g.stride_b % 2 == 0);
    a.tiles_m = a.tiles_n = 0;
    auto tiles = [&](int bm, int bn) { return ((g.M + bm - 1) / bm) * ((g.N + bn - 1) / bn) * g.batch; };
    const double c64 = tiling_cost(tiles(64, 64), 64 * 64, 33.4);
    const double c64x32 = tiling_cost(tiles(64, 32), 64 * 32, 30.9);
    const double c32 = tiling_cost(tiles(32, 32), 32 * 32, 29.3);
    if (c64 <= c64x32 && c64 <= c32) return launch_layout<64, 64, 32, 32>(g, a, stream);
    if (c64x32 <= c32) return launch_layout<64, 32, 32, 16>(g, a, stream);
    return launch_layout<32, 32, 16, 16>(g, a, stream);
}

}  // namespace gatlas
