"""GEMV where the column blocks of the cluster kernel change width (floats 32, 64,
32, 128 columns; doubles 32, 64, 32, 64), at the first and last columns of each
range, a segment's ends, and the switch to the general kernel; and the image
engine, which runs the same kernels below its own sizes.  Integers small enough
that every order of summation is exact."""
import numpy as np
import pytest

import gatlas_b200 as g

pytestmark = pytest.mark.gpu

# widths change after 1472, 12800, 14208 and 25600 columns (float), 4096, 18944
# and 28416 (double) on 148 SMs; 1300 x 10240 doubles take the general kernel
COLUMNS = [(1152, 515), (1472, 64), (1476, 513), (4096, 130), (4100, 131), (12800, 65), (12804, 64), (14208, 33),
           (14212, 70), (18944, 64), (18948, 129), (25600, 40), (25604, 66), (28416, 9), (28420, 64), (1300, 10239),
           (1300, 10240)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("M,N", COLUMNS)
def test_columns_exact(cuda, dtype, M, N):
    import torch
    rng = np.random.default_rng(M + N)
    A = rng.integers(-3, 4, M * N).astype(dtype)
    x = rng.integers(-3, 4, N).astype(dtype)
    y0 = rng.integers(-9, 10, M).astype(dtype)
    want = 2 * (A.reshape(N, M).T.astype(np.float64) @ x.astype(np.float64)) - y0
    dA, dx = torch.from_numpy(A).to(cuda), torch.from_numpy(x).to(cuda)
    for engine in ("buffer", "image"):
        y = torch.from_numpy(y0.copy()).to(cuda)
        g.matvec(dA, dx, M, N, y=y, trans_a=True, gemv=True, alpha=2.0, beta=-1.0, engine=engine)
        assert np.array_equal(y.cpu().numpy(), want.astype(dtype)), engine
    assert g.device_faults() == 0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
# a lane's vectors 1, 4, 5, 7 and 8 with warps that end inside a group, row counts
# where a warp's rows change; long rows in whole and in part
@pytest.mark.parametrize("M,N", [(1, 4), (17, 4096), (2372, 1000), (9474, 64), (6808, 516), (6812, 508), (11844, 260),
                                 (14212, 132), (37, 7168), (37, 7200), (39, 8192), (41, 8196), (5, 20484)])
def test_image_rows_exact(cuda, dtype, M, N):
    import torch
    rng = np.random.default_rng(M + N)
    A = rng.integers(-3, 4, M * N).astype(dtype)
    x = rng.integers(-3, 4, N).astype(dtype)
    y = g.matvec(torch.from_numpy(A).to(cuda), torch.from_numpy(x).to(cuda), M, N, engine="image").cpu().numpy()
    assert np.array_equal(y, (A.reshape(M, N).astype(np.float64) @ x.astype(np.float64)).astype(dtype))


def test_image_refusals_hold(cuda):
    """A workspace smaller than the query's answer, or off 256 bytes, is refused
    also where the product would not use it."""
    import torch
    M = N = 1024
    A, x = (torch.zeros(s, device=cuda) for s in (M * N, N))
    need = g.matvec_workspace_size(M, N, trans_a=True)
    buf = torch.empty(need + 512, dtype=torch.uint8, device=cuda)
    buf = buf[(-buf.data_ptr()) % 256:]
    d = g.matvec_desc(M, N, trans_a=True, engine="image")
    y = torch.empty(M, device=cuda)
    import ctypes

    def call(ptr, size):
        return g.lib().gatlas_matvec_f32(ctypes.byref(d), A.data_ptr(), x.data_ptr(), y.data_ptr(), ptr, size,
                                         torch.cuda.current_stream().cuda_stream)
    assert call(buf.data_ptr(), need) == 0
    assert call(buf.data_ptr(), 16) != 0
    assert call(buf.data_ptr() + 16, need) != 0
