"""GEMV at the sizes where its kernels, tails and cluster splits change: both
layouts, float and double, with and without 16-byte aligned rows, within the
normwise tolerance 4*N*u of the FP64 product, and exactly where every product
and sum is exact."""
import numpy as np
import pytest

import gatlas_b200 as g
import oracle

pytestmark = pytest.mark.gpu
U = {np.float32: 2.0 ** -24, np.float64: 2.0 ** -53}


def _run(cuda, A, x, M, N, ta, yin=None, **kw):
    import torch
    y = None if yin is None else torch.from_numpy(yin.copy()).to(cuda)
    return g.matvec(torch.from_numpy(A).to(cuda), torch.from_numpy(x).to(cuda), M, N, y=y, trans_a=ta, **kw).cpu().numpy()


# row-major: lengths around 4 x 256 and 8 x 256 loads of one element and 4 x 256
# of a vector, few and many rows; column-major: widths around the least for
# clusters, the change of block width, 1, 2, 4 and 8 segments, ragged segments
SIZES = [(3, 1023), (700, 1024), (5000, 1025), (9, 2047), (301, 2050), (33, 4095), (2, 4097), (1201, 4100),
         (591, 63), (592, 129), (609, 700), (1025, 517), (2048, 1000), (2049, 999), (4096, 64), (4099, 131),
         (9000, 300), (20001, 40), (24000, 333)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("M,N", SIZES)
def test_within_tolerance(cuda, dtype, ta, M, N):
    A = oracle.uniform(M * N, seed=M + N, dtype=dtype)
    x = oracle.uniform(N, seed=N, dtype=dtype)
    yin = oracle.uniform(M, seed=M, dtype=dtype)
    a = A.reshape(N, M).T if ta else A.reshape(M, N)
    exact = a.astype(np.longdouble) @ x.astype(np.longdouble)
    bar = 4 * N * U[dtype] * float(np.linalg.norm((np.abs(a.astype(np.float64)) @ np.abs(x.astype(np.float64)))))
    y = _run(cuda, A, x, M, N, ta)
    assert float(np.linalg.norm((y - exact).astype(np.float64))) <= bar
    y = _run(cuda, A, x, M, N, ta, yin, gemv=True, alpha=0.5, beta=-2.0)
    assert float(np.linalg.norm((y - (0.5 * exact - 2 * yin.astype(np.longdouble))).astype(np.float64))) <= bar


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("M,N", [(1201, 4099), (640, 2051), (5003, 1030)])
def test_exact_sums_and_batch(cuda, ta, M, N):
    """Small integers: every order of summation gives the same exact result."""
    rng = np.random.default_rng(M)
    P = 2
    A = rng.integers(-3, 4, P * M * N).astype(np.float32)
    x = rng.integers(-3, 4, P * N).astype(np.float32)
    y = _run(cuda, A, x, M, N, ta, batch=P).reshape(P, M)
    for p in range(P):
        a = A[p * M * N:(p + 1) * M * N]
        a = a.reshape(N, M).T if ta else a.reshape(M, N)
        assert np.array_equal(y[p], (a.astype(np.float64) @ x[p * N:(p + 1) * N].astype(np.float64)).astype(np.float32))


@pytest.mark.parametrize("ta", [0, 1])
def test_infinities_stay_in_their_rows(cuda, ta):
    M, N = 643, 1027
    A, x = np.ones(M * N, np.float32), np.ones(N, np.float32)
    a = A.reshape(N, M).T if ta else A.reshape(M, N)
    a[642, 1026], a[5, 0] = np.inf, np.nan
    y = _run(cuda, A, x, M, N, ta)
    want = np.full(M, float(N), np.float32)
    want[642], want[5] = np.inf, np.nan
    assert np.array_equal(y, want, equal_nan=True)
