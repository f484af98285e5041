"""The one-launch tensor-core contraction (products of few tiles, no caller
workspace) against the two-pass path (caller's workspace): bit for bit, since
both run the same pieces through the same MMA sequence."""
import ctypes

import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu
ENGINES = ["tc_bf16", "tc_split3", "tc_split6"]


def _aligned(cuda, nbytes):
    import torch
    buf = torch.empty(nbytes + 1024, dtype=torch.uint8, device=cuda)
    return buf[-buf.data_ptr() % 1024:]


def _uniform(cuda, n, seed):
    import torch
    return g.fill(torch.empty(n, dtype=torch.float32, device=cuda), "uniform", seed=seed)


def _both(cuda, engine, M, N, K, ta, tb, alpha=1.0, beta=0.0, batch=1, A=None, B=None):
    import torch
    A = _uniform(cuda, batch * M * K, M + K) if A is None else A
    B = _uniform(cuda, batch * K * N, N + K) if B is None else B
    C0 = _uniform(cuda, batch * M * N, 5) if beta else torch.full((batch * M * N,), float("nan"), device=cuda)
    ws = _aligned(cuda, g.matmul_workspace_size(M, N, K, engine, ta, tb, batch))
    kw = dict(trans_a=ta, trans_b=tb, gemm=True, alpha=alpha, beta=beta, engine=engine, batch=batch)
    one = g.matmul(A, B, M, N, K, C=C0.clone(), **kw).cpu().numpy()
    two = g.matmul(A, B, M, N, K, C=C0.clone(), workspace=ws, **kw).cpu().numpy()
    assert g.device_faults() == 0
    return one, two


# tile edges (64 and 128 rows, 32 and 64 columns), remainders of a 64-deep slice
# and of a 16-byte vector, segments of one and several slices, one slice only
@pytest.mark.parametrize("engine", ENGINES)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 33, 64), (65, 31, 63), (128, 64, 260), (130, 200, 1001),
                                   (50, 70, 2051), (700, 900, 333), (1000, 1000, 100)])
def test_same_bits_as_two_passes(cuda, engine, ta, tb, M, N, K):
    one, two = _both(cuda, engine, M, N, K, ta, tb)
    assert np.array_equal(one, two)


@pytest.mark.parametrize("engine", ENGINES)
@pytest.mark.parametrize("batch", [1, 3])
def test_alpha_beta_and_instances(cuda, engine, batch):
    one, two = _both(cuda, engine, 100, 75, 190, 0, 1, alpha=0.75, beta=-1.5, batch=batch)
    assert np.array_equal(one, two)


@pytest.mark.parametrize("engine", ENGINES)
def test_infinities_and_nan(cuda, engine):
    import torch
    M, N, K = 70, 40, 150
    A, B = _uniform(cuda, M * K, 1), _uniform(cuda, K * N, 2)
    A.view(M, K)[3, 5], A.view(M, K)[69, 149], B.view(K, N)[7, 39] = float("inf"), float("nan"), float("-inf")
    one, two = _both(cuda, engine, M, N, K, 0, 0, A=A, B=B)
    assert np.array_equal(one, two, equal_nan=True)


@pytest.mark.parametrize("engine,extra", [("tc_bf16", 1), ("tc_bf16", 3), ("tc_split3", 1), ("tc_split3", 7),
                                          ("tc_split6", 1), ("tc_split6", 2), ("tc_split6", 6)])
def test_promotion_intervals(cuda, engine, extra):
    """Intervals of one slice and of more segments than TMEM buffers; an odd
    split6 interval (slices of 32) takes the two-pass path."""
    import torch
    M, N, K = 90, 96, 1400
    A, B = _uniform(cuda, M * K, 3), _uniform(cuda, K * N, 4)
    ws = _aligned(cuda, g.matmul_workspace_size(M, N, K, engine))
    tile = (0, 0, 0, 0, 0, extra)
    one = g.matmul(A, B, M, N, K, engine=engine, tile=tile)
    two = g.matmul(A, B, M, N, K, engine=engine, tile=tile, workspace=ws)
    assert torch.equal(one, two) and g.device_faults() == 0


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad,off", [(1, 0), (4, 0), (4, 1)])
def test_leading_dimensions_and_bases(cuda, ta, tb, pad, off):
    """Rows padded to odd and to 16-byte lengths, bases on and off a 16-byte
    boundary; C's padding and the gap between instances stay untouched."""
    import torch
    M, N, K, P = 70, 45, 130, 2
    a_rows, a_in = (K, M) if ta else (M, K)
    b_rows, b_in = (N, K) if tb else (K, N)
    lda, ldb, ldc = a_in + pad, b_in + pad, N + pad
    sa, sb, sc = a_rows * lda + 4 * pad, b_rows * ldb + 4 * pad, M * ldc + pad
    A, B, C = (_uniform(cuda, P * s + off, s)[off:] for s in (sa, sb, sc))
    C1 = C.clone()
    d = g.matmul_desc(M, N, K, ta, tb, True, 0.5, 2.0, "tc_split3", batch=P, lda=lda, ldb=ldb, ldc=ldc, stride_a=sa,
                      stride_b=sb, stride_c=sc)
    need = int(g.lib().gatlas_matmul_workspace_size(ctypes.byref(d)))
    ws = _aligned(cuda, need)
    for out, w in ((C, None), (C1, ws)):
        g.check(g.lib().gatlas_matmul_f32(ctypes.byref(d), A.data_ptr(), B.data_ptr(), out.data_ptr(),
                                          None if w is None else w.data_ptr(), 0 if w is None else need,
                                          torch.cuda.current_stream().cuda_stream))
    assert torch.equal(C, C1) and g.device_faults() == 0


@pytest.mark.parametrize("engine,bar", [("tc_bf16", 2.0 ** -7), ("tc_split3", 8e-6), ("tc_split6", 2.5e-6)])
def test_error_against_the_oracle(cuda, engine, bar):
    M, N, K = 48, 100, 1030
    A, B = oracle.uniform(M * K, seed=1), oracle.uniform(K * N, seed=2)
    import torch
    C = g.matmul(torch.from_numpy(A).to(cuda), torch.from_numpy(B).to(cuda), M, N, K, engine=engine).cpu().numpy()
    ref = A.reshape(M, K).astype(np.float64) @ B.reshape(K, N).astype(np.float64)
    assert oracle.normwise_error(C, ref.ravel()) <= bar
