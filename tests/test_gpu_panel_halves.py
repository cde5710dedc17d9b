"""GPU: LU panels of more than 12,288 rows, which a cluster eliminates in two halves of 32 columns.

Planted factors with small integers and eighths, so that every step is exact in FP32: unit lower L with entries below
1, U with powers of two on the diagonal, rows shuffled.  The largest candidate of each column is then unique and the
panel has to give back the permutation and both factors bit for bit, in the left half, in the right half's update and in
the rows that the right half's interchanges move.  Sizes: the smallest and largest row counts of each number of rows
per thread, with remainders.
"""
import ctypes

import pytest
import torch

from updes_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12289, 16384, 16401, 20480, 20500, 24576])
def test_planted_panel(n):
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    L = torch.randint(-7, 8, (n, 64), generator=g, device="cuda").double() / 8
    L[:64] = torch.tril(L[:64], -1) + torch.eye(64, device="cuda", dtype=torch.float64)
    U = torch.triu(torch.randint(-3, 4, (64, 64), generator=g, device="cuda").double(), 1)
    U += torch.diag(torch.where(torch.rand(64, generator=g, device="cuda") < 0.5, 8.0, -4.0).double())
    perm = torch.randperm(n, generator=g, device="cuda")
    ld = int(lib.updes_matrix_ld(n, 8))
    A = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    A[:, :64] = L @ U
    d = torch.arange(64, n, device="cuda")
    A[d, d] = 2.0
    A = A[perm].contiguous()
    F = torch.zeros((n, ld), dtype=torch.float32, device="cuda")
    piv = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    nb, info = ctypes.c_size_t(), ctypes.c_int32(-1)
    _lib.check(lib.updes_lu_workspace(n, 1, ctypes.byref(nb)), "updes_lu_workspace")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.updes_lu_factor(n, A.data_ptr(), ld, 1, F.data_ptr(), ld, piv.data_ptr(), ws.data_ptr(),
                                   ws.numel(), ctypes.byref(info), s), "updes_lu_factor")
    torch.cuda.synchronize()
    assert info.value == 0
    rows = perm.cpu().tolist()
    for k, p in enumerate(piv[:n].cpu().tolist()):
        assert k <= p < n
        rows[k], rows[p] = rows[p], rows[k]
    assert rows == list(range(n))
    want = L.clone()
    want[:64] = torch.tril(L[:64], -1) + U
    assert torch.equal(F[:, :64].double(), want)
    assert torch.equal(torch.diagonal(F[64:, 64:n]).double(), torch.full((n - 64,), 2.0, device="cuda", dtype=torch.float64))
