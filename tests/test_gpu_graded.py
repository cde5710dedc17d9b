"""GPU: the FP64 paths on matrices whose rows and columns are of very different size.  A collocation matrix of r^(2a+1) on
a domain of side S has kernel entries of S^(2a+1) beside the ones of its polynomial block."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nodes(nx, ny, side):
    rng = np.random.default_rng(nx * ny)
    ids = np.arange(nx * ny)
    ii, jj = ids // ny, ids % ny
    X = np.stack([np.linspace(0.0, 1.0, nx)[ii], np.linspace(0.0, 1.0, ny)[jj]], axis=-1)
    inner = (ii > 0) & (ii < nx - 1) & (jj > 0) & (jj < ny - 1)
    X[inner] += rng.uniform(-0.2, 0.2, size=(nx * ny, 2))[inner] * min(1.0 / (nx - 1), 1.0 / (ny - 1))
    return X * side


def _lu(A):
    import torch
    from updes_gb300 import _lib
    lib = _lib.load()
    n = A.shape[0]
    ld = int(lib.updes_matrix_ld(n, 8))
    F = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    F[:, :n] = torch.as_tensor(A)
    piv = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    nb, info = ctypes.c_size_t(), ctypes.c_int32(-1)
    _lib.check(lib.updes_lu_workspace(n, _lib.PREC_FP64, ctypes.byref(nb)), "updes_lu_workspace")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    _lib.check(lib.updes_lu_factor(n, F.data_ptr(), ld, _lib.PREC_FP64, F.data_ptr(), ld, piv.data_ptr(), ws.data_ptr(),
                                   ws.numel(), ctypes.byref(info),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "updes_lu_factor")
    assert info.value == 0
    LU, PA = F.cpu().numpy()[:, :n], A[piv.cpu().numpy()[n:]]
    return PA, np.tril(LU, -1) + np.eye(n), np.triu(LU)


def _graded(kind, n):
    if kind == "rows":
        rng = np.random.default_rng(n)
        return rng.standard_normal((n, n)) * 2.0 ** rng.integers(-60, 60, (n, 1))
    nx, ny = (n - 3) // 20, 20
    X = _nodes(nx, ny, 2.0 ** -10)
    r = np.sqrt(((X[:, None] - X[None]) ** 2).sum(-1))
    P = np.concatenate([np.ones((len(X), 1)), X], axis=1)
    return np.block([[r ** (3 if kind == "r3" else 5), P], [P.T, np.zeros((3, 3))]])


@pytest.mark.parametrize("kind,n", [("rows", 33), ("rows", 300), ("rows", 1100), ("r3", 603), ("r5", 403), ("r3", 1203)])
def test_lu_factor_takes_any_scaling(kind, n):
    # a chain of multiply-adds per entry: |PA - LU| <= n u |L||U|, and the check's own product once more
    A = _graded(kind, n)
    PA, L, U = _lu(A)
    wrong = np.abs(PA - L @ U) > 2 * A.shape[0] * 2.0 ** -53 * (np.abs(L) @ np.abs(U))
    assert not wrong.any(), f"{int(wrong.sum())} entries"
