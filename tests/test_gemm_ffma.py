"""The float default point (asynchronous copies, tile by size) against the
sequential fma chain: bit for bit at tile edges and remainders of each tiling,
every layout, padded and odd leading dimensions, packed instances, and inputs
with infinities, NaN and signed zeros."""
import ctypes

import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu


def _gpu(cuda, a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _same(C, ref):
    assert np.array_equal(C, ref, equal_nan=True)
    assert np.array_equal(np.signbit(C[ref == 0]), np.signbit(ref[ref == 0]))


# 32 x 32, 64 x 64, 128 x 64 and 128 x 128 tiles are chosen for the groups of sizes
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (33, 31, 17), (96, 80, 16), (257, 130, 101),
                                   (1100, 1099, 35), (1025, 1000, 33), (2049, 2047, 17)])
def test_bit_exact(cuda, ta, tb, M, N, K):
    A = oracle.uniform(M * K, seed=M + K, dtype=np.float32)
    B = oracle.uniform(K * N, seed=N + K, dtype=np.float32)
    C = g.matmul(_gpu(cuda, A), _gpu(cuda, B), M, N, K, trans_a=ta, trans_b=tb).cpu().numpy()
    _same(C, oracle.matmul(A, B, M, N, K, ta, tb, mode=oracle.FMA, dtype=np.float32))


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
@pytest.mark.parametrize("pad", [1, 4])
def test_leading_dimensions_and_instances(cuda, ta, tb, pad):
    """Odd padding and 16-byte rows (4- and 16-byte copies), two instances with a gap."""
    import torch
    M, N, K, P = 72, 48, 40, 2
    a_rows, a_in = (K, M) if ta else (M, K)
    b_rows, b_in = (N, K) if tb else (K, N)
    lda, ldb, ldc = a_in + pad, b_in + pad, N + pad
    sa, sb, sc = a_rows * lda + 4 * pad, b_rows * ldb + 4 * pad, M * ldc + pad
    A, B, C0 = (oracle.uniform(P * s, seed=s, dtype=np.float32) for s in (sa, sb, sc))
    C = _gpu(cuda, C0)
    d = g.matmul_desc(M, N, K, ta, tb, True, 0.75, -1.25, "buffer", batch=P, lda=lda, ldb=ldb, ldc=ldc, stride_a=sa,
                      stride_b=sb, stride_c=sc)
    dA, dB = _gpu(cuda, A), _gpu(cuda, B)
    g.check(g.lib().gatlas_matmul_f32(ctypes.byref(d), dA.data_ptr(), dB.data_ptr(), C.data_ptr(), None, 0,
                                      torch.cuda.current_stream().cuda_stream))
    want = C0.copy()
    for p in range(P):
        a = A[p * sa:p * sa + a_rows * lda].reshape(a_rows, lda)[:, :a_in].ravel()
        b = B[p * sb:p * sb + b_rows * ldb].reshape(b_rows, ldb)[:, :b_in].ravel()
        c = want[p * sc:p * sc + M * ldc].reshape(M, ldc)
        c[:, :N] = oracle.matmul(np.ascontiguousarray(a), np.ascontiguousarray(b), M, N, K, ta, tb, mode=oracle.FMA,
                                 gemm=1, Cin=np.ascontiguousarray(c[:, :N]).ravel(), alpha=0.75, beta=-1.25,
                                 dtype=np.float32).reshape(M, N)
    _same(C.cpu().numpy(), want)


def test_special_values(cuda):
    M, N, K = 40, 48, 21
    rng = np.random.default_rng(3)
    A, B = (rng.standard_normal(n).astype(np.float32) for n in (M * K, K * N))
    for x in (A, B):
        x[rng.integers(0, x.size, 60)] = rng.choice([np.inf, -np.inf, np.nan, 0.0, -0.0, 1e-45, 3e38], 60)
    A.reshape(M, K)[3] = -0.0
    C = g.matmul(_gpu(cuda, A), _gpu(cuda, B), M, N, K).cpu().numpy()
    _same(C, oracle.matmul(A, B, M, N, K, mode=oracle.FMA, dtype=np.float32))


def test_empty_contraction_scales_c(cuda):
    M, N = 65, 33
    C0 = oracle.uniform(M * N, seed=2, dtype=np.float32)
    e = _gpu(cuda, np.zeros(0, np.float32))
    C = g.matmul(e, e, M, N, 0, C=_gpu(cuda, C0), gemm=True, alpha=1.0, beta=0.5).cpu().numpy()
    assert np.array_equal(C, 0.5 * C0)
