"""GPU: the panels' pivots where they are decided by rule: exact ties in later panels, between rows of different CTAs that
earlier interchanges have renumbered, and what follows a column without a pivot."""
import numpy as np
import pytest

from test_gpu_panel import _factor, _reconstruct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [150, 800, 1500])
def test_ties_in_every_panel(n, precision):
    # Rows u_i of an upper triangular matrix of small integers with 2 on its diagonal, to one of which, for each column j,
    # +-u_j has been added, in any order.  Step j chooses between the two rows that hold +-2 there; whichever goes first
    # leaves +-u_i of the other, so every step is exact and LAPACK's rule, the first of them, decides all pivots.
    from scipy.linalg import lapack
    rng = np.random.default_rng(n)
    U = 2.0 * np.eye(n)
    A, free = np.zeros((n, n)), list(range(1, n))
    for j in range(n - 1):
        U[j, rng.integers(j + 1, n, 3)] = rng.choice([-1.0, 1.0], 3)
    A += U
    for j in range(n - 1):
        later = [i for i in free if i > j]
        if later:
            i = later[rng.integers(len(later))]
            free.remove(i)
            A[i] += rng.choice([-1.0, 1.0]) * U[j]
    A = A[rng.permutation(n)]
    _, want, _ = lapack.dgetrf(A)
    st, info, F, piv = _factor(A, precision)
    assert st == 0 and info == 0
    assert np.array_equal(piv.cpu().numpy()[:n], want)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,column", [(400, 70), (400, 255), (1100, 300)])
def test_what_follows_a_zero_column(n, column, precision):
    rng = np.random.default_rng(n + column)
    A = rng.standard_normal((n, n))
    A[:, column] = 0.0
    st, info, F, piv = _factor(A, precision)
    assert info == column + 1
    PA, L, U, p = _reconstruct(A, F, piv)
    assert np.all(p >= np.arange(n)) and np.all(p < n)
    assert np.array_equal(np.sort(piv.cpu().numpy()[n:]), np.arange(n))
    assert np.isfinite(L).all() and np.isfinite(U).all() and np.all(U[:, column] == 0.0) and np.max(np.abs(L)) <= 1 + 2.0 ** -22
    # FP64: a chain of multiply-adds per entry, and the check's own; mixed: as without the zero column, 64 FP32 roundings
    bound = 2 * n * 2.0 ** -53 if precision == 0 else 64 * 2.0 ** -24
    wrong = np.abs(PA - L @ U) > bound * (np.abs(L) @ np.abs(U))
    assert not wrong.any(), f"{int(wrong.sum())} entries"
