"""FP8 products that CTA pairs or single CTAs may serve, as the device decides
from the lengths of the segments: either way the bits of the forced tilings."""
import numpy as np
import pytest

import gatlas_b200 as g
from captured import kernel_names

pytestmark = pytest.mark.gpu


def _operand(rng, rows, K, varied):
    """Block magnitudes 2^-3 .. 2^3: all alike, changing with every block of K, or
    changing in every other block row."""
    kb = -(-K // 128)
    e = rng.integers(-3, 4, (-(-rows // 128), kb))
    if varied == "none":
        e[:] = 0
    elif varied == "half":
        e[::2] = 0
    x = rng.uniform(-1, 1, (rows, K)).astype(np.float32)
    return x * np.exp2(e).astype(np.float32).repeat(128, 0)[:rows].repeat(128, 1)[:, :K]


# more than 148 blocks of 256 x 256, last ones partial; 8 blocks of K at least
@pytest.mark.parametrize("M,N,K", [(3201, 3101, 1030), (257, 37900, 1100)])
@pytest.mark.parametrize("varied", ["none", "half", "all"])
def test_same_bits_as_the_forced_tilings(cuda, M, N, K, varied):
    import torch
    rng = np.random.default_rng(M + K)
    a, b = _operand(rng, M, K, varied), _operand(rng, N, K, "none" if varied == "half" else varied)
    A, B = (torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in (a, b))
    C = torch.empty(M * N, device=cuda)
    run = lambda: g.matmul(A, B, M, N, K, C=C, trans_b=True, engine="tc_fp8")  # noqa: E731
    got = []
    try:
        for pair in (0, 2):
            g.set_option("tc_pair", pair)
            C.fill_(float("nan"))
            run()
            got.append(C.clone())
    finally:
        g.set_option("tc_pair", 1)
    names = kernel_names(run)  # quantisation, plan and both contractions
    assert len(names) == 4 and sum("tc_gemm_persistent_kernel" in n for n in names) == 2
    C.fill_(float("nan"))
    run()
    assert torch.equal(C, got[0]) and torch.equal(C, got[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
        run()
    C.fill_(float("nan"))
    graph.replay()
    assert torch.equal(C, got[0]) and g.device_faults() == 0


# one less than 8 blocks of K, and too few tiles: one contraction
@pytest.mark.parametrize("M,N,K", [(3201, 3101, 896), (1000, 3000, 1100)])
def test_small_products_run_on_single_ctas(cuda, M, N, K):
    import torch
    A, B = torch.ones(M * K, device=cuda), torch.ones(N * K, device=cuda)
    C = torch.empty(M * N, device=cuda)
    names = kernel_names(lambda: g.matmul(A, B, M, N, K, C=C, trans_b=True, engine="tc_fp8"))
    assert len(names) == 3 and "Li3ELb0E" in names[2]
    g.matmul(A, B, M, N, K, C=C, trans_b=True, engine="tc_fp8")
    assert bool((C == K).all())


# row blocks of 512 (the last partial): single CTAs, or blocks wide enough for either
@pytest.mark.parametrize("M,N,K", [(2300, 700, 1500), (1100, 19200, 1030)])
def test_host_pipeline_on_varied_scales(cuda, M, N, K):
    """Each row block contracts with its own part of the plan."""
    import torch
    rng = np.random.default_rng(M)
    A, B = (torch.from_numpy(np.ascontiguousarray(_operand(rng, r, K, "all")).ravel()) for r in (M, N))
    want = g.matmul(A.to(cuda), B.to(cuda), M, N, K, trans_b=True, engine="tc_fp8").cpu()
    C = torch.full((M * N,), float("nan")).pin_memory()
    g.matmul_host(A.pin_memory(), B.pin_memory(), M, N, K, C, trans_b=True, engine="tc_fp8")
    torch.cuda.synchronize()
    assert g.device_faults() == 0
    assert torch.equal(C, want)
