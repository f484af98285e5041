"""C = alpha AB + beta C of the default SIMT points: the epilogue's batched
reads of C against the sequential fma chain, bit for bit, where tiles are
ragged in rows, in whole vectors of columns and in single columns, with 16-byte
and narrower rows of C."""
import ctypes

import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("M,N", [(31, 28), (33, 37), (130, 260), (257, 131), (900, 904), (1100, 1102), (2049, 2052)])
def test_update_bit_exact(cuda, dtype, pad, M, N):
    import torch
    K, ldc = 19, N + pad
    A = oracle.uniform(M * K, seed=M, dtype=dtype)
    B = oracle.uniform(K * N, seed=N, dtype=dtype)
    C0 = oracle.uniform(M * ldc, seed=3, dtype=dtype)
    dA, dB, C = (torch.from_numpy(x.copy()).to(cuda) for x in (A, B, C0))
    d = g.matmul_desc(M, N, K, False, True, True, 0.75, -1.25, "buffer", ldc=ldc)
    fn = g.lib().gatlas_matmul_f32 if dtype == np.float32 else g.lib().gatlas_matmul_f64
    g.check(fn(ctypes.byref(d), dA.data_ptr(), dB.data_ptr(), C.data_ptr(), None, 0,
               torch.cuda.current_stream().cuda_stream))
    got = C.cpu().numpy().reshape(M, ldc)
    Cin = np.ascontiguousarray(C0.reshape(M, ldc)[:, :N]).ravel()
    want = oracle.matmul(A, B, M, N, K, 0, 1, mode=oracle.FMA, gemm=1, Cin=Cin, alpha=0.75, beta=-1.25, dtype=dtype)
    assert np.array_equal(got[:, :N].ravel(), want)
    assert np.array_equal(got[:, N:], C0.reshape(M, ldc)[:, N:])
