"""GPU: the LU panels at the sizes where their split over threads, CTAs and clusters changes: rows around a CTA's
256 and 512, clusters of 1 to 16, widths below a full panel, repeated and unusable pivots."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import lu_factor_random

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 63, 64, 65, 255, 256, 257, 513, 769, 1025, 2049, 4097]


def _reconstruct(A, F, piv):
    n = A.shape[0]
    LU = F.cpu().numpy()[:, :n].astype(np.float64)
    p = piv.cpu().numpy()
    PA = A.copy()
    for k in range(n):
        if p[k] != k:
            PA[[k, p[k]]] = PA[[p[k], k]]
    L = np.tril(LU, -1) + np.eye(n)
    U = np.triu(LU)
    return PA, L, U, p[:n]


@pytest.mark.parametrize("n", SIZES)
def test_mixed_panel_backward_error(n):
    A, F, _, piv, _, _ = lu_factor_random(n, 1, n)
    PA, L, U, p = _reconstruct(A, F, piv)
    assert np.all(p >= np.arange(n)) and np.all(p < n)
    # a panel's own columns are eliminated in FP32, at most 64 updates an entry: 64 * 2^-24 of |L||U|
    assert np.all(np.abs(PA - L @ U) <= 64 * 2.0 ** -24 * (np.abs(L) @ np.abs(U)))
    assert np.max(np.abs(L)) <= 1 + 2.0 ** -22  # the multipliers of a partial pivoting, rounded in FP32


@pytest.mark.parametrize("n", SIZES + [1100, 1281, 2400])
def test_fp64_lu(n):
    from scipy.linalg import lapack
    A, F, _, piv, _, _ = lu_factor_random(n, 0, n)
    PA, L, U, p = _reconstruct(A, F, piv)
    _, want, _ = lapack.dgetrf(A)
    assert np.array_equal(p, want)
    # the trailing updates (at most n / 256 + 12 of an entry) cut each operand at 2^-56 of a power of two up to twice
    # its row's (column's) largest entry and leave out products that sum to at most 2^-43 of the two largest ones in
    # the worst case; the panels and triangular solves round like FP64 arithmetic
    worst = np.max(np.abs(L), axis=1)[:, None] * np.max(np.abs(U), axis=0)[None, :]
    assert np.all(np.abs(PA - L @ U) <= (n / 256 + 12) * 2.0 ** -43 * worst + n * 2.0 ** -53 * (np.abs(L) @ np.abs(U)))
    # and on random data it is as good as LAPACK's own factors
    lu, _, _ = lapack.dgetrf(A)
    ref = np.linalg.norm(PA - (np.tril(lu, -1) + np.eye(n)) @ np.triu(lu))
    assert np.linalg.norm(PA - L @ U) <= 4 * ref + 1e-300


def test_fp64_update_scales():
    # rows and columns of very different size, exact zeros and a zero row, against LAPACK column by column
    from scipy.linalg import lapack
    rng = np.random.default_rng(3)
    n = 700
    A = rng.standard_normal((n, n)) * 2.0 ** rng.integers(-300, 300, n)[None, :]
    A[rng.random((n, n)) < 0.3] = 0.0
    st, info, F, piv = _factor(A, 0)
    assert st == 0 and info == 0
    PA, L, U, p = _reconstruct(A, F, piv)
    scale = np.max(np.abs(A), axis=0)
    assert np.max(np.abs((PA - L @ U) / scale)) <= 1e-12


def _factor(A, precision):
    import torch
    from updes_gb300 import _lib
    lib = _lib.load()
    n = A.shape[0]
    ld = int(lib.updes_matrix_ld(n, 8))
    Ad = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    Ad[:, :n] = torch.as_tensor(A)
    F = torch.zeros((n, ld), dtype=torch.float32, device="cuda") if precision else Ad
    piv = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    nb = ctypes.c_size_t()
    _lib.check(lib.updes_lu_workspace(n, precision, ctypes.byref(nb)), "updes_lu_workspace")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    info = ctypes.c_int32(-1)
    st = lib.updes_lu_factor(n, Ad.data_ptr(), ld, precision, F.data_ptr() if precision else Ad.data_ptr(), ld,
                             piv.data_ptr(), ws.data_ptr(), ws.numel(), ctypes.byref(info),
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return st, info.value, F, piv


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [65, 300, 800])
def test_ties_take_the_first_row(n, precision):
    # small integers: every step exact, many rows share the largest entry; LAPACK's rule is the first of them
    from scipy.linalg import lapack
    rng = np.random.default_rng(n)
    A = np.triu(rng.integers(1, 3, (n, n)).astype(np.float64))
    A[n // 2:, 0] = A[0, 0]          # column 0: ties between row 0 and the lower half
    A[n // 3, :] = A[0, :] * 1.0     # and equal rows leave zeros that never become pivots
    A[n // 3, n // 3] += 4.0
    _, want, _ = lapack.dgetrf(A)
    st, info, F, piv = _factor(A, precision)
    assert np.array_equal(piv.cpu().numpy()[:n][:8], want[:8])


@pytest.mark.parametrize("precision", [0, 1])
def test_zero_column_reports_its_step_and_goes_on(precision):
    rng = np.random.default_rng(5)
    n = 400
    A = rng.standard_normal((n, n))
    A[:, 70] = 0.0
    st, info, F, piv = _factor(A, precision)
    assert info == 71
