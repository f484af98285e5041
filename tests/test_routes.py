"""Kernels that only some sizes reach, each at sizes where it can go wrong
(tile and vector remainders), with the kernel that ran named: the library
chooses by size, and a test of one kernel must not run another."""
import pytest

import gatlas_b200 as g
from captured import kernel_names

pytestmark = pytest.mark.gpu


def _uniform(cuda, n, seed):
    import torch
    return g.fill(torch.empty(n, dtype=torch.float32, device=cuda), "uniform", seed=seed)


# Operands off the 16-byte grid (odd K), over many 64-deep slices, so that the
# ring and the warp groups turn; against the two-pass path bit for bit.
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("engine,M,N,K", [("tc_bf16", 64, 50, 501), ("tc_bf16", 130, 200, 251),
                                          ("tc_split3", 40, 70, 1501), ("tc_split3", 130, 200, 501),
                                          ("tc_split6", 64, 100, 3001), ("tc_split6", 130, 200, 2051)])
def test_one_launch_contraction_of_unaligned_operands(cuda, engine, ta, tb, M, N, K):
    import torch
    A, B = _uniform(cuda, M * K, 1), _uniform(cuda, K * N, 2)
    one = torch.full((M * N,), float("nan"), device=cuda)
    two = torch.full((M * N,), float("nan"), device=cuda)
    size = g.matmul_workspace_size(M, N, K, engine, ta, tb)
    buf = torch.empty(size + 1024, dtype=torch.uint8, device=cuda)
    ws = buf[-buf.data_ptr() % 1024:]
    kw = dict(trans_a=ta, trans_b=tb, engine=engine)
    names = kernel_names(lambda: g.matmul(A, B, M, N, K, C=one, **kw))
    assert len(names) == 1 and "tc_gemm_direct_kernel" in names[0]
    names = kernel_names(lambda: g.matmul(A, B, M, N, K, C=two, workspace=ws, **kw))
    assert len(names) == 2 and not any("direct" in n for n in names)
    g.matmul(A, B, M, N, K, C=one, **kw)
    g.matmul(A, B, M, N, K, C=two, workspace=ws, **kw)
    assert g.device_faults() == 0
    assert torch.equal(one, two)


# Several waves of tiles re-reading large operands: the split pass is cheaper.
@pytest.mark.parametrize("engine,M,N,K,batch,ta,tb", [("tc_bf16", 16, 3688, 3320, 7, 1, 1),
                                                      ("tc_split3", 2580, 152, 2588, 8, 1, 0)])
def test_large_operands_are_split_first(cuda, engine, M, N, K, batch, ta, tb):
    import torch
    A, B = _uniform(cuda, batch * M * K, 1), _uniform(cuda, batch * K * N, 2)
    C = torch.empty(batch * M * N, device=cuda)
    names = kernel_names(lambda: g.matmul(A, B, M, N, K, C=C, trans_a=ta, trans_b=tb, engine=engine, batch=batch))
    assert len(names) == 2 and "split_kernel" in names[0]


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
