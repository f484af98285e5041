"""The split pass of the two-pass tensor-core path, both operands in one launch:
at the edges of its work blocks (512 runs of eight k, 64 x 64 tiles), with whole
and partial runs, aligned and unaligned rows, several instances.  Products of few
tiles without a workspace split their operands inside the contraction, with code
of its own, and run the same products in the same order: results are compared bit
for bit."""
import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["tc_bf16", "tc_split3", "tc_split6"])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K,batch", [(1, 1, 1, 1), (64, 64, 64, 1), (65, 63, 64, 1), (512, 8, 8, 2), (513, 40, 7, 1),
                                         (3, 5, 4104, 1), (127, 129, 65, 3), (100, 36, 1000, 1)])
def test_two_passes_match_the_direct_contraction(cuda, engine, ta, tb, M, N, K, batch):
    import torch
    A = torch.from_numpy(oracle.uniform(M * K * batch, seed=M + K)).to(cuda)
    B = torch.from_numpy(oracle.uniform(K * N * batch, seed=N + K)).to(cuda)
    direct = g.matmul(A, B, M, N, K, trans_a=ta, trans_b=tb, engine=engine, batch=batch).cpu().numpy()
    buf = torch.empty(g.matmul_workspace_size(M, N, K, engine, ta, tb, batch=batch) + 1024, dtype=torch.uint8, device=cuda)
    ws = buf[(-buf.data_ptr()) % 1024:]
    two = g.matmul(A, B, M, N, K, trans_a=ta, trans_b=tb, engine=engine, batch=batch, workspace=ws).cpu().numpy()
    assert g.device_faults() == 0
    assert np.array_equal(direct.view(np.uint32), two.view(np.uint32))
