"""GPU: the FP64 triangular solves (L, U and their transposes) around their blocks of 64 and halves of 32."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import lu_factor_random
from updes_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 200, 321])
def test_fp64_triangular_solves(n, trans):
    import torch
    lib = _lib.load()
    A, F, ld, piv, ws, s = lu_factor_random(n, 0, 3 * n + trans)
    LU = F.cpu().numpy()[:, :n]
    perm = piv.cpu().numpy()[n:2 * n]
    b = np.random.default_rng(n).standard_normal(n)
    x = torch.as_tensor(b, device="cuda").clone().reshape(n, 1)
    _lib.check(lib.updes_lu_solve(n, F.data_ptr(), ld, 0, piv.data_ptr(), x.data_ptr(), 1, 1, trans, ws.data_ptr(),
                                  ws.numel(), s), "updes_lu_solve")
    torch.cuda.synchronize()
    x = x[:, 0].cpu().numpy().astype(np.longdouble)
    L = (np.tril(LU, -1) + np.eye(n)).astype(np.longdouble)
    U = np.triu(LU).astype(np.longdouble)
    # L U x = P b, or (L U)^T P x = b: each substitution leaves a residual of at most (n + 3) roundoffs of |T||x| (two more
    # than plain substitution for the rows scaled by reciprocals), the two together at most twice that of |L||U||x|
    if trans:
        y = x[perm]
        res = U.T @ (L.T @ y) - b
        size = np.abs(U.T) @ (np.abs(L.T) @ np.abs(y))
    else:
        res = L @ (U @ x) - b[perm]
        size = np.abs(L) @ (np.abs(U) @ np.abs(x))
    assert np.all(np.abs(res) <= 2 * (n + 3) * 2.0 ** -52 * size)
