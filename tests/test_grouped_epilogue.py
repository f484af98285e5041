"""The grouped contraction's epilogue at each access width: 16, 8 and 4 bytes a
lane, by the multiple that every instance's N and leading dimension share.  Same
products in the same order as the single-instance engine, one fused multiply-add
per element of C: results are compared bit for bit, and nothing outside the N
columns of a row is written."""
import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["tc_bf16", "tc_split3"])
@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("width", [4, 2, 1])
def test_epilogue_widths(cuda, engine, pair, width):
    import torch
    # (m, n / width, k, pad / width, gemm, alpha, beta): chunk and tile edges, idle
    # column parts, a tile of one row, all of -0.0 and beta = -0.0
    shapes = [(1, 1, 3, 0, 1, 0.5, 1.0), (31, 8, 64, 1, 1, 2.0, 1.0), (33, 9, 40, 0, 0, 1.0, 0.0),
              (128, 33, 65, 3, 1, -1.0, -0.0), (129, 64, 17, 0, 1, 1.0, 0.5), (257, 65, 130, 1, 1, 0.0, -0.0)]
    inst, host = [], []
    for i, (m, nw, k, pad, gemm, alpha, beta) in enumerate(shapes):
        n, ldc = nw * width, (nw + pad) * width
        A, B = oracle.uniform(m * k, seed=7 * i + 1), oracle.uniform(k * n, seed=7 * i + 2)
        C0 = oracle.uniform(m * ldc, seed=7 * i + 3)
        host.append((C0, m, n, ldc))
        inst.append(dict(A=torch.from_numpy(A).to(cuda), B=torch.from_numpy(B).to(cuda),
                         C=torch.from_numpy(C0.copy()).to(cuda), m=m, n=n, k=k, ldc=ldc, gemm=gemm, alpha=alpha,
                         beta=beta))
    old = g.get_option("grouped_pair")
    g.set_option("grouped_pair", pair)
    try:
        plan = g.Grouped(inst, engine=engine)
        plan.prepare().run()
        got = [q["C"].cpu().numpy().copy() for q in inst]
        for q, h in zip(inst, host):
            q["C"].copy_(torch.from_numpy(h[0]))
        plan.run_each()
        want = [q["C"].cpu().numpy().copy() for q in inst]
        plan.close()
    finally:
        g.set_option("grouped_pair", old)
    assert g.device_faults() == 0
    for x, y, (C0, m, n, ldc) in zip(got, want, host):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (m, n)
        assert np.array_equal(x.reshape(m, ldc)[:, n:], C0.reshape(m, ldc)[:, n:])
