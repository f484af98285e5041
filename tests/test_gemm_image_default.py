"""The image engine's default point, which runs the faster of its own and the
buffer engine's default kernel: the same bits as an explicit point of its own on
both sides of that choice, every layout, padded rows, packed instances, and the
same refusals."""
import ctypes

import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu


def _run(cuda, dtype, A, B, C0, M, N, K, ta, tb, tile, **ld):
    import torch
    dA, dB, C = (torch.from_numpy(x).to(cuda) for x in (A, B, C0))
    d = g.matmul_desc(M, N, K, ta, tb, True, 0.75, -1.25, "image", tile=tile, **ld)
    fn = g.lib().gatlas_matmul_f32 if dtype == np.float32 else g.lib().gatlas_matmul_f64
    g.check(fn(ctypes.byref(d), dA.data_ptr(), dB.data_ptr(), C.data_ptr(), None, 0,
               torch.cuda.current_stream().cuda_stream))
    out = C.cpu().numpy()
    assert g.device_faults() == 0
    return out


# 1536 x 1532 x 1024 with A transposed stays on tensor maps in float; the rest do not
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K,P", [(4, 4, 4, 1), (132, 100, 36, 2), (1536, 1532, 1024, 1), (1536, 1532, 1020, 1)])
def test_same_bits_as_an_explicit_point(cuda, dtype, ta, tb, M, N, K, P):
    pad = 4
    a_rows, a_in = (K, M) if ta else (M, K)
    b_rows, b_in = (N, K) if tb else (K, N)
    ld = dict(lda=a_in + pad, ldb=b_in + pad, ldc=N + 1, batch=P)
    ld.update(stride_a=a_rows * ld["lda"] + 4, stride_b=b_rows * ld["ldb"] + 4, stride_c=M * ld["ldc"] + 3)
    A, B, C0 = (oracle.uniform(P * s, seed=s, dtype=dtype) for s in (ld["stride_a"], ld["stride_b"], ld["stride_c"]))
    args = (cuda, dtype, A, B, C0, M, N, K, ta, tb)
    tile = (16, 16, 8, 8, 0) if dtype == np.float32 else (16, 16, 4, 4, 0)
    assert np.array_equal(_run(*args, None, **ld), _run(*args, tile, **ld))


@pytest.mark.parametrize("dtype,K", [(np.float32, 30), (np.float64, 31)])
def test_unaligned_rows_stay_refused(cuda, dtype, K):
    M = N = 64
    A, B, C0 = (oracle.uniform(s, seed=s, dtype=dtype) for s in (M * K, K * N, M * N))
    with pytest.raises(RuntimeError, match="16-byte"):
        _run(cuda, dtype, A, B, C0, M, N, K, 0, 0, None)
