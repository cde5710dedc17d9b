"""GPU: the batched right-hand-side solve and the prepared values at the sizes where their tiles change: below, at and
above 64-row blocks, 128-row and 256-wide digit blocks, and column groups of 8, against LAPACK on the assembled system."""
import ctypes

import numpy as np
import pytest

import updes_gb300 as U
from gpu_helpers import assemble
from updes_gb300 import _lib
from updes_gb300.multirhs import MultiRHSSolver
from updes_gb300.operators import _interp_problem

pytestmark = pytest.mark.gpu

FACETS = {"South": "d", "West": "d", "North": "d", "East": "d"}
# n = Nx Ny + 3: 12, 63, 65, 127, 129, 255, 259, 515
GRIDS = [(3, 3), (10, 6), (31, 2), (31, 4), (42, 3), (42, 6), (16, 16), (32, 16)]


def _op(x, center, rbf, monomial, fields=None):
    return U.nodal_value(x, center, rbf, monomial) - 0.01 * U.nodal_laplacian(x, center, rbf, monomial)


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("R", [1, 7, 8, 9, 64])
def test_blocks_match_lapack(nx, ny, R):
    import torch
    cloud = U.SquareCloud(Nx=nx, Ny=ny, facet_types=FACETS)
    bcs = {f: np.zeros(len(cloud.facet_nodes[f])) for f in FACETS}
    s = MultiRHSSolver(_op, cloud, bcs, U.polyharmonic, 1)
    K = assemble(s.dp)[0].cpu().numpy()[:, :s.n]
    A = assemble(_interp_problem(cloud, U.polyharmonic, 1))[0].cpu().numpy()[:s.N, :s.n]
    rng = np.random.default_rng(nx * 100 + R)
    want = rng.standard_normal((s.n, R))
    Q = K[:s.N] @ want
    # the polynomial rows of the right-hand side are zero: solve for what that system holds
    want = np.linalg.solve(K, np.vstack([Q, np.zeros((s.n - s.N, R))]))
    C, V = s.solve(Q)
    # the residual uses K rounded to 2^-48 an entry and refinement settles within its condition number of that
    tol = 64 * np.linalg.cond(K) * 2.0 ** -48 + 1e-13
    C = C.cpu().numpy()
    assert np.linalg.norm(C - want) <= tol * np.linalg.norm(want)
    # values of given coefficients: each of at most 3 k blocks rounded once, operands cut at 2^-56 of the largest entry of
    # a row (column) in a k block of at most 256 entries
    Vp = V.cpu().numpy()
    bound = 256 * 2.0 ** -54 * np.max(np.abs(A), axis=1)[:, None] * np.max(np.abs(C), axis=0)[None, :] + \
        2.0 ** -50 * (np.abs(A) @ np.abs(C))
    assert np.all(np.abs(Vp - A @ C) <= bound + 2.0 ** -50 * (np.abs(A) @ np.abs(C)))


def test_prepared_values_equal_plain_ones():
    import torch
    lib = _lib.load()
    cloud = U.SquareCloud(Nx=23, Ny=17, facet_types=FACETS)
    bcs = {f: np.zeros(len(cloud.facet_nodes[f])) for f in FACETS}
    s = MultiRHSSolver(_op, cloud, bcs, U.polyharmonic, 1)
    C = torch.as_tensor(np.random.default_rng(0).standard_normal((s.n, 5)), device="cuda")
    V, W = (torch.empty((s.N, 5), dtype=torch.float64, device="cuda") for _ in range(2))
    s._eval_into(C, V, s.dp.stream())
    _lib.check(lib.updes_eval_values_batch(ctypes.byref(s.dp.c), 5, C.data_ptr(), 5, W.data_ptr(), 5, s.dp.stream()),
               "updes_eval_values_batch")
    assert torch.max(torch.abs(V - W)).item() <= 1e-13 * torch.max(torch.abs(W)).item()


def test_values_without_a_preparation_are_nan():
    import torch
    cloud = U.SquareCloud(Nx=9, Ny=9, facet_types=FACETS)
    bcs = {f: np.zeros(len(cloud.facet_nodes[f])) for f in FACETS}
    s = MultiRHSSolver(_op, cloud, bcs, U.polyharmonic, 1)
    s.bws.zero_()
    C = torch.ones((s.n, 2), dtype=torch.float64, device="cuda")
    V = torch.zeros((s.N, 2), dtype=torch.float64, device="cuda")
    s._eval_into(C, V, s.dp.stream())
    assert torch.isnan(V).all()
