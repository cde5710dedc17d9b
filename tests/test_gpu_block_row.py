"""GPU: the block row of U of the mixed LU around the CTAs of 16 columns (1 to 17 and more columns beside the first block
of 256 rows) and on both sides of the 8,192 columns up to which one kernel forms it."""
import numpy as np
import pytest
import torch

from gpu_helpers import lu_factor_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [257, 258, 271, 272, 273, 289, 520, 8447, 8448, 8449])
def test_backward_error(n):
    A, F, _, piv, _, _ = lu_factor_random(n, 1, n + 2)
    LU = F[:, :n].double()
    rows = torch.as_tensor(piv.cpu().numpy()[n:2 * n].astype(np.int64), device="cuda")
    PA = torch.as_tensor(A, device="cuda")[rows]
    x = torch.as_tensor(np.random.default_rng(n).standard_normal((n, 3)), device="cuda")
    L, U = torch.tril(LU, -1), torch.triu(LU)
    y = U @ x
    res = PA @ x - (L @ y + y)
    size = L.abs() @ (U.abs() @ x.abs()) + U.abs() @ x.abs()
    # a panel's own columns are eliminated in FP32, at most 64 updates an entry: 64 * 2^-24 of |L||U|
    assert bool(torch.all(res.abs() <= 64 * 2.0 ** -24 * size))
    assert float(torch.linalg.norm(res) / torch.linalg.norm(size)) <= 2.0 ** -24
