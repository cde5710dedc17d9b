"""GPU: values, gradients and Laplacians of polyharmonic fields (the FP32-seeded root and the shortened sums) against 64-bit
NumPy: points on centers, distances down to 2^-30 and far outside the root's FP32 range, ragged counts."""
import numpy as np
import pytest

import updes_gb300 as U
from functools import partial

pytestmark = pytest.mark.gpu


def _exact(P, C, c, a, what):
    d = P[:, None].astype(np.longdouble) - C[None].astype(np.longdouble)
    r2 = (d ** 2).sum(-1)
    r = np.sqrt(r2)
    k = 2 * a + 1
    lam = c[:len(C)].astype(np.longdouble)
    if what == 0:
        t = r ** k
    elif what == 1:
        t = k * r ** (k - 2)
        return np.stack([(t * d[..., i]) @ lam for i in (0, 1)], -1), np.stack(
            [np.abs(t * d[..., i]) @ np.abs(lam) for i in (0, 1)], -1)
    else:
        t = k * k * r ** (k - 2)
    return t @ lam, np.abs(t) @ np.abs(lam)


@pytest.mark.parametrize("a", [1, 2, 3])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -30, 2.0 ** 30, 2.0 ** -45, 2.0 ** 45])
@pytest.mark.parametrize("m,N", [(1, 1), (7, 33), (65, 512), (33, 515)])
def test_polyharmonic_fields(a, scale, m, N):
    rng = np.random.default_rng(m * 1000 + N + a)
    C = rng.uniform(0, 1, (N, 2))
    P = rng.uniform(0, 1, (m, 2))
    P[::3] = C[rng.integers(0, N, len(P[::3]))]                       # on a center
    P[1::3] = C[rng.integers(0, N, len(P[1::3]))] + 2.0 ** -30        # next to one
    C, P = C * scale, P * scale
    c = np.concatenate([rng.standard_normal(N), np.zeros(3)])
    rbf = partial(U.polyharmonic, a=a)
    for what, fn in enumerate((U.value_vec, U.gradient_vec, U.laplacian_vec)):
        got = np.asarray(fn(P, c, C, rbf))
        want, size = _exact(P, C, c, a, what)
        # differences, r^2, the root, at most a + 3 products: 2a + 10 roundings a term, and a sum of N terms
        tol = (2 * a + 10 + 4 * np.sqrt(N)) * 2.0 ** -53
        assert np.all(np.abs(got - want) <= tol * size), (what, np.max(np.abs(got - want) / np.maximum(size, 1e-300)))
