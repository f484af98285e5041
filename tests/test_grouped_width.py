"""Access width to C of a grouped plan whose rows are off the 16-byte grid: pairs,
or single floats where C is written only and larger than L2; either way the
bits of the single-instance engine."""
import pytest

import gatlas_b200 as g
from captured import kernel_names

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,betas,width", [(33, 0.0, 1), (32, 0.0, 2), (33, 0.5, 2)])
def test_width_follows_size_and_beta(cuda, count, betas, width):
    import torch
    m, n, k = 1024, 1022, 33  # 33 products hold more than 2^25 elements of C, 32 fewer

    def rand(size, seed):
        return g.fill(torch.empty(size, device=cuda), "uniform", seed=seed)

    inst = [dict(A=rand(m * k, i), B=rand(k * n, 100 + i), C=rand(m * n, 200 + i), m=m, n=n, k=k, gemm=1, alpha=0.5,
                 beta=betas if i == count - 1 else 0.0) for i in range(count)]
    start = [q["C"].clone() for q in inst]
    plan = g.Grouped(inst, engine="tc_bf16")
    plan.prepare()
    names = kernel_names(plan.run)
    assert len(names) == 1 and f"grouped_gemm_kernelILi0ELb0ELi{width}EE" in names[0], names

    def result(run):
        for q, c in zip(inst, start):
            q["C"].copy_(c)
        run()
        return [q["C"].clone() for q in inst]

    assert all(torch.equal(x, y) for x, y in zip(result(plan.run), result(plan.run_each)))
    assert g.device_faults() == 0
    plan.close()
