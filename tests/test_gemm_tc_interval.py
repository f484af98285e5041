"""The promotion interval (the descriptor's extra) at the ends of its range:
counts above the number of K slices accumulate all of K, counts of 2^31 and
above are the default, on the one-launch and the two-pass path alike."""
import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu
LARGEST = 2 ** 31 - 1


def _product(cuda, engine, M, N, K, extra, workspace):
    import torch
    A = torch.from_numpy(oracle.uniform(M * K, seed=1)).to(cuda)
    B = torch.from_numpy(oracle.uniform(K * N, seed=2)).to(cuda)
    ws = None
    if workspace:
        size = g.matmul_workspace_size(M, N, K, engine)
        buf = torch.empty(size + 1024, dtype=torch.uint8, device=cuda)
        ws = buf[-buf.data_ptr() % 1024:]
    C = torch.full((M * N,), float("nan"), device=cuda)
    g.matmul(A, B, M, N, K, C=C, engine=engine, tile=(0, 0, 0, 0, 0, extra), workspace=ws)
    assert g.device_faults(clear=True) == 0
    return C.cpu().numpy()


# (64 rows run in one launch without a workspace, 300 x 600 in two passes)
@pytest.mark.parametrize("engine", ["tc_bf16", "tc_split3", "tc_split6", "tc_fp8"])
@pytest.mark.parametrize("M,N", [(64, 96), (300, 600)])
@pytest.mark.parametrize("workspace", [False, True])
def test_intervals_at_the_ends_of_the_range(cuda, engine, M, N, workspace):
    K = 1100
    default = _product(cuda, engine, M, N, K, 0, workspace)
    for extra in (2 ** 31, 2 ** 32 - 2, 2 ** 32 - 1):
        assert np.array_equal(_product(cuda, engine, M, N, K, extra, workspace), default)
    # all of K: at least as many slices as there are (K <= 2048 in any slice depth of 32 or more)
    whole = _product(cuda, engine, M, N, K, 64, workspace)
    for extra in (LARGEST - 1, LARGEST):
        assert np.array_equal(_product(cuda, engine, M, N, K, extra, workspace), whole)
    assert np.array_equal(whole, _product(cuda, engine, M, N, K, 64, not workspace))


@pytest.mark.parametrize("ta,tb", [(1, 1), (0, 0), (0, 1)])
def test_depth_beyond_the_transposing_split_is_refused_either_way(cuda, ta, tb):
    """An operand stored across k is split in a grid of 65535 tiles of 64 k; with
    and without a workspace the answer is the same (both along k: accepted)."""
    import torch
    K = 65535 * 64 + 8
    A, B = torch.ones(K, device=cuda), torch.ones(K, device=cuda)
    size = g.matmul_workspace_size(1, 1, K, "tc_split3", ta, tb)
    buf = torch.empty(size + 1024, dtype=torch.uint8, device=cuda)
    for ws in (None, buf[-buf.data_ptr() % 1024:]):
        if ta or not tb:
            with pytest.raises(g.GatlasError, match="too large"):
                g.matmul(A, B, 1, 1, K, trans_a=ta, trans_b=tb, engine="tc_split3", workspace=ws)
        else:
            C = g.matmul(A, B, 1, 1, K, trans_a=ta, trans_b=tb, engine="tc_split3", workspace=ws)
            assert abs(float(C) - K) <= 2.0 ** -24 * K * (K // 256) ** 0.5
