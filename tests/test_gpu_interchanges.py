"""GPU: the permutation that the factorisation leaves behind its interchanges is the one they compose to, at sizes
around the groups of four and the CTAs of 128 positions that build it."""
import numpy as np
import pytest

from gpu_helpers import lu_factor_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 64, 127, 128, 129, 131, 256, 385, 1101])
def test_permutation_of_the_interchanges(n, precision):
    *_, piv, _, _ = lu_factor_random(n, precision, 5 * n + 1)
    p = piv.cpu().numpy()
    want = np.arange(n)
    for k in range(n):
        want[[k, p[k]]] = want[[p[k], k]]
    assert np.array_equal(p[n:2 * n], want)
