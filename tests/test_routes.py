"""Kernels that only some sizes reach, each at sizes where it can go wrong
(tile and vector remainders), with the kernel that ran named: the library
chooses by size, and a test of one kernel must not run another."""
import pytest

import gatlas_b200 as g
from captured import kernel_names

pytestmark = pytest.mark.gpu


def _matvec_exact(cuda, engine, M, N, dtype, trans_a, kernel):
    """Small integers, so that every order of summation gives the same bits."""
    import torch
    dt = getattr(torch, dtype)
    gen = torch.Generator(device=cuda).manual_seed(M + N)
    A = torch.randint(-3, 4, (M * N,), generator=gen, device=cuda, dtype=torch.int8).to(dt)
    x = torch.randint(-3, 4, (N,), generator=gen, device=cuda, dtype=torch.int8).to(dt)
    y0 = torch.randint(-3, 4, (M,), generator=gen, device=cuda, dtype=torch.int8).to(dt)
    y = y0.clone()
    kw = dict(trans_a=trans_a, gemv=True, alpha=2.0, beta=-3.0, engine=engine)
    names = kernel_names(lambda: g.matvec(A, x, M, N, y=y, **kw))
    assert len(names) == 1 and kernel in names[0], names
    y.copy_(y0)
    g.matvec(A, x, M, N, y=y, **kw)
    assert g.device_faults() == 0
    product = torch.zeros(M, dtype=torch.float64, device=cuda)
    rows = N if trans_a else M
    inner = M if trans_a else N
    for i in range(0, rows, 4096):
        part = A[i * inner:min(i + 4096, rows) * inner].view(-1, inner).double()
        if trans_a:
            product += part.t() @ x[i:i + 4096].double()
        else:
            product[i:i + 4096] = part @ x.double()
    assert torch.equal(y.double(), 2.0 * product - 3.0 * y0.double())


# TMA tiles: 16 rows x 256 floats or 128 doubles (rows), 32 rows x 128 doubles
# (columns); last row block, last chunk and last segment partial
@pytest.mark.parametrize("M,N,dtype", [(1700, 20004, "float32"), (4420, 15408, "float32"), (1601, 8002, "float64"),
                                       (4730, 8002, "float64")])
def test_image_rows_on_tiles(cuda, M, N, dtype):
    _matvec_exact(cuda, "image", M, N, dtype, False, "gemv_rows_tma_kernel")


@pytest.mark.parametrize("M,N", [(17452, 580), (2530, 21470), (130, 1001), (2, 33)])
def test_image_columns_on_tiles(cuda, M, N):
    _matvec_exact(cuda, "image", M, N, "float64", True, "gemv_cols_tma_kernel")


# rows that end 1 vector, and just under and over 1.25 vectors a thread, after
# whole groups of 1024; doubles in few and in many rows
@pytest.mark.parametrize("M,N,dtype,kernel", [
    (301, 4100, "float32", "gemv_rowblock_kernelIfLi4ELi2ELi4ELb1E"),
    (301, 5372, "float32", "gemv_rowblock_kernelIfLi4ELi2ELi4ELb1E"),
    (301, 5376, "float32", "gemv_rowblock_kernelIfLi4ELi2ELi4ELb0E"),
    (33, 8196, "float32", "gemv_rowblock_kernelIfLi4ELi2ELi4ELb0E"),
    (33, 8194, "float64", "gemv_rowblock_kernelIdLi2ELi2ELi4ELb1E"),
    (33, 17402, "float64", "gemv_rowblock_kernelIdLi2ELi2ELi4ELb1E"),
    (1801, 4098, "float64", "gemv_rowblock_kernelIdLi2ELi2ELi4ELb1E"),
    (1801, 8194, "float64", "gemv_rowblock_kernelIdLi2ELi2ELi4ELb0E"),
    (4001, 2342, "float32", "gemv_rows_kernelIfLi1E"),
    (7105, 2343, "float64", "gemv_rows_kernelIdLi1ELi2E"),
    (4739, 1025, "float64", "gemv_rows_kernelIdLi1ELi2E"),
    (9473, 4501, "float32", "gemv_rows_kernelIfLi1ELi2E"),
    (9473, 3501, "float32", "gemv_rows_kernelIfLi1ELi2E"),
    (301, 3501, "float32", "gemv_rowblock_kernelIfLi1E")])
def test_buffer_rows(cuda, M, N, dtype, kernel):
    _matvec_exact(cuda, "buffer", M, N, dtype, False, kernel)


# every column-cluster kernel, with a last block and a last segment that are not
# whole, and one row more than a segment takes
@pytest.mark.parametrize("M,N,dtype,kernel", [
    (600, 1025, "float32", "cluster_kernelIfLb1ELi8E"),
    (1540, 2051, "float32", "cluster_kernelIfLb1ELi16E"),
    (12804, 1029, "float32", "cluster_kernelIfLb1ELi32E"),
    (601, 1537, "float32", "cluster_kernelIfLb0ELi16ELi2E"),
    (2371, 2049, "float32", "cluster_kernelIfLb0ELi16ELi4E"),
    (15001, 1027, "float32", "cluster_kernelIfLb0ELi16ELi4E"),
    (5001, 8199, "float32", "cluster_kernelIfLb0ELi32ELi2E"),
    (1030, 771, "float64", "cluster_kernelIdLb1ELi16ELi2ELi8ELi2ELi5E"),
    (4200, 2049, "float64", "cluster_kernelIdLb1ELi32E"),
    (24002, 513, "float64", "cluster_kernelIdLb1ELi16ELi2ELi8ELi2ELi6E")])
def test_column_clusters(cuda, M, N, dtype, kernel):
    _matvec_exact(cuda, "buffer", M, N, dtype, True, kernel)
