"""GPU: the mixed LU's tensor-core updates recover planted factors bit for bit.

A = L U with 64 x 64 diagonal blocks of L the identity and of U diagonal (powers of two), so that the panels and the
triangular solves compute nothing that could round.  Off those blocks one factor has 23-bit entries, the other small
integers: every product and every sum of an update fits the double-float pair and the update's accumulators, and every
digit of the 23-bit factor takes part.  The diagonal is the largest entry of each column, so no row moves.
Sizes: trailing matrices of 1 to 897 rows and columns, around the tiles of 64 and 128 and with odd remainders; 1,153 has
the look-ahead.
"""
import ctypes

import numpy as np
import pytest
import torch

from updes_gb300 import _lib

pytestmark = pytest.mark.gpu


def _factor(A):
    lib, n = _lib.load(), len(A)
    ld = int(lib.updes_matrix_ld(n, 8))
    Ad = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    Ad[:, :n] = torch.as_tensor(A)
    F = torch.zeros((n, ld), dtype=torch.float32, device="cuda")
    piv = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    nb, info = ctypes.c_size_t(), ctypes.c_int32(-1)
    _lib.check(lib.updes_lu_workspace(n, 1, ctypes.byref(nb)), "updes_lu_workspace")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.updes_lu_factor(n, Ad.data_ptr(), ld, 1, F.data_ptr(), ld, piv.data_ptr(), ws.data_ptr(),
                                   ws.numel(), ctypes.byref(info), s), "updes_lu_factor")
    torch.cuda.synchronize()
    assert info.value == 0
    return F[:, :n].cpu().numpy().astype(np.float64), piv[:n].cpu().numpy()


@pytest.mark.parametrize("fine", ["L", "U"])
@pytest.mark.parametrize("n", [257, 319, 320, 321, 384, 385, 449, 641, 1153])
def test_planted_factors(n, fine):
    rng = np.random.default_rng(n)
    many = rng.integers(-(1 << 23) + 1, 1 << 23, (n, n)) / float(1 << 23)
    few = rng.integers(-7, 8, (n, n)) / 8.0
    Lx, Ux = (many, 8.0 * few) if fine == "L" else (few, 8.0 * many)
    off = (np.arange(n)[:, None] // 64) != (np.arange(n)[None, :] // 64)
    L = np.tril(Lx, -1) * off + np.eye(n)
    U = np.triu(Ux, 1) * off + np.diag(np.where(rng.integers(0, 2, n) > 0, 8.0, -4.0))
    F, piv = _factor(L @ U)  # exact in FP64: 23 + 4 bits and up to 1,153 terms
    assert np.array_equal(piv, np.arange(n))
    assert np.array_equal(np.tril(F, -1) + np.eye(n), L)
    assert np.array_equal(np.triu(F), U)
