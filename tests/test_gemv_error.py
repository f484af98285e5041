"""Rounding error of column-major GEMV against 64 bits: no larger than that of
rows cut into four CTAs' segments per SM, whatever the kernel that runs.

Bar: summing L values one after the other adds about 0.4 * 2^-24 * sqrt(L / 2)
of the result's norm (each addition rounds by 0.4 ulp rms of a partial sum that
grows as sqrt(i)), and lengths add up over the levels of a sum in parts.  With
148 SMs, blocks of 128 columns and 8 warps a block's levels are its rows per
warp, the 8 warps and its segments.  Too strict by 0 to 12 % on those sums
themselves (it leaves out the final rounding)."""
import math

import numpy as np
import pytest

import gatlas_b200 as g

pytestmark = pytest.mark.gpu


def _bar(M, N):
    blocks = -(-M // 128)
    segments = max(1, min(-(-592 // blocks), -(-N // 32)))
    rows = -(-N // segments)
    segments = -(-N // rows)
    return 0.4 * 2.0 ** -24 * math.sqrt((rows / 8 + 8 + segments) / 2)


# every cluster shape: 64 columns with 1, 2 and 8 segments, 128 columns, 32
# columns, and rows off the 16-byte grid with 32 and 64
@pytest.mark.parametrize("engine", ["buffer", "image"])
@pytest.mark.parametrize("M,N", [(16384, 16384), (20000, 6000), (12000, 10000), (60000, 500), (25600, 4096),
                                 (2048, 2048), (1024, 32768), (2047, 12001), (5001, 14003)])
def test_column_major_error(cuda, engine, M, N):
    import torch
    if engine == "image" and M % 4:
        pytest.skip("16-byte rows only")
    A = g.fill(torch.empty(M * N, dtype=torch.float32, device=cuda), "uniform", seed=M)
    x = g.fill(torch.empty(N, dtype=torch.float32, device=cuda), "uniform", seed=N)
    y = g.matvec(A, x, M, N, trans_a=True, engine=engine).double()
    exact = torch.zeros(M, dtype=torch.float64, device=cuda)
    for j in range(0, N, 1024):
        rows = min(1024, N - j)
        exact += A[j * M:(j + rows) * M].view(rows, M).double().t() @ x[j:j + rows].double()
    err = float((y - exact).norm() / exact.norm())
    assert err <= _bar(M, N)
