"""FP8 segment plans: every tiling promotes at the same blocks of K, so single
CTAs, CTA pairs and the default give the same bits whatever the block scales."""
import numpy as np
import pytest

import gatlas_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(129, 300, 5000), (640, 257, 4096), (1000, 1000, 1300), (2560, 2304, 260)])
@pytest.mark.parametrize("extra", [0, 1, 3])
def test_tilings_agree_on_varied_scales(cuda, M, N, K, extra):
    """Block magnitudes vary by powers of two in runs of random length (more
    than 32 blocks of K in the first case: several words of the plan)."""
    import torch
    rng = np.random.default_rng(M + N + K)

    def operand(rows):
        blocks = np.repeat(rng.integers(-3, 4, (-(-rows // 128), 200)), rng.integers(1, 4, 200), axis=1)[:, :-(-K // 128)]
        x = rng.uniform(-1, 1, (rows, K)).astype(np.float32)
        return x * np.exp2(blocks).astype(np.float32).repeat(128, 0)[:rows].repeat(128, 1)[:, :K]

    a, b = operand(M), operand(N)
    A, B = (torch.from_numpy(np.ascontiguousarray(v).ravel()).to(cuda) for v in (a, b))
    got = []
    try:
        for pair in (0, 1, 2):
            g.set_option("tc_pair", pair)
            got.append(g.matmul(A, B, M, N, K, trans_b=True, engine="tc_fp8", tile=(0, 0, 0, 0, 0, extra)).cpu().numpy())
    finally:
        g.set_option("tc_pair", 1)
    assert g.device_faults() == 0
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    ref = a.astype(np.float64) @ b.astype(np.float64).T
    assert np.linalg.norm(got[0].reshape(M, N) - ref) <= 2.0 ** -4 * np.linalg.norm(ref)
