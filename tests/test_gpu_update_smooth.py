"""GPU: the mixed LU's trailing update on rows and columns that hardly vary, whose remainders add up with one sign.

A = [[I, U], [L, L U + T]] with FP32 L and U: 256 steps leave L and U as they are and T, the update's result, as the matrix
still to be factored, whose first row is the factor's and whose first column is L's times the pivot."""
import numpy as np
import pytest

from test_gpu_panel import _factor

pytestmark = pytest.mark.gpu

K, M = 256, 700  # one update of 256 steps, tiles of 128 and a remainder


def _operands(kind):
    rng = np.random.default_rng(4)
    L = np.repeat(rng.uniform(0.5, 1.0, (M, 1)), K, axis=1)
    U = np.repeat(rng.uniform(0.5, 1.0, (1, M)), K, axis=0)
    k = np.arange(K)
    if kind == "slow":      # 2^-10 over the row: less than a leading digit
        L, U = L * (1.0 - k / (1024.0 * K)), U * (1.0 - k / (1024.0 * K))[:, None]
    elif kind == "smooth":  # a kernel's decay along a row
        L, U = L * np.exp(-k / K), U * np.exp(-2.0 * k / K)[:, None]
    elif kind == "signs":   # and without a common sign
        L, U = L * np.where(k % 3, 1.0, -1.0), U * np.where(k % 2, 1.0, -1.0)[:, None]
    return L.astype(np.float32).astype(np.float64), U.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("kind", ["constant", "slow", "smooth", "signs"])
def test_update_of_rows_that_hardly_vary(kind):
    L, U = _operands(kind)
    rng = np.random.default_rng(7)
    T = np.round(rng.uniform(0.25, 0.5, (M, M)) * 2.0 ** 20) / 2.0 ** 20
    T[0, 0] = 2.0
    wide = np.longdouble
    P = np.zeros((M, M), wide)
    for k in range(K):
        P += np.outer(L[:, k].astype(wide), U[k].astype(wide))
    A = np.block([[np.eye(K), U], [L, (P + T).astype(np.float64)]])
    st, info, F, piv = _factor(A, 1)
    F = F.cpu().numpy()[:, :K + M].astype(np.float64)
    p = piv.cpu().numpy()
    assert st == 0 and info == 0 and np.array_equal(p[:K + 1], np.arange(K + 1))
    rows = p[K + M:][K + 1:] - K  # T's rows in the factors' order
    # Each of the 32 instructions that add to g1 may drop 2^-32 of |L||U| (remainders of one sign), 2^-27 in all; and the FP32
    # roundings of what is read: half a unit of 2^-25 in the row, and of a quotient and a half by a pivot of 2 in the column.
    size = np.abs(L) @ np.abs(U)
    row, column = np.abs(F[K, K + 1:] - T[0, 1:]), np.abs(F[K + 1:, K] * 2.0 - T[rows, 0])
    assert np.max(row - 2.0 ** -27 * size[0, 1:]) <= 2.0 ** -26
    assert np.max(column - 2.0 ** -27 * size[rows, 0]) <= 2.0 ** -24
