"""GPU: the refinement's fused Gram-Schmidt passes and residual at sizes around their 120 chunks (fewer unknowns than
chunks, one more, a remainder) and with restart lengths that end cycles after one, two or many vectors.

The reported convergence is checked against values of the FP64 factorisation: the mixed solve stops at a backward error
of at most 256 roundoffs (or 1e-13 of ||b||), FP64 LU at a few; on these systems (condition below 1e5) the two agree to
1e-8 of the largest value."""
from functools import partial

import numpy as np
import pytest

import updes_gb300 as U
from updes_gb300 import operators as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [1, 2, 40])
@pytest.mark.parametrize("shape", [(3, 3), (10, 10), (9, 13), (11, 11), (12, 20), (20, 18)])
def test_mixed_against_fp64(shape, restart):
    cloud = U.SquareCloud(Nx=shape[0], Ny=shape[1], facet_types={f: "d" for f in ("North", "South", "West", "East")})
    bcs = {f: (lambda c: 1.0 + c[0] * c[1]) for f in ("North", "South", "West", "East")}
    args = dict(diff_operator=lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial),
                rhs_operator=lambda x, centers, rbf, fields: np.cos(3 * x[0]) * x[1], cloud=cloud,
                boundary_conditions=O.boundary_conditions_func_to_arr(bcs, cloud),
                rbf=partial(U.polyharmonic, a=1), max_degree=1)
    want = U.pde_solver(**args, options=U.SolverOptions(precision="fp64", reuse_factorization=False)).vals
    got = U.pde_solver(**args, options=U.SolverOptions(precision="fp32", restart=restart, fallback_fp64=False,
                                                       reuse_factorization=False)).vals
    info = dict(O.LAST_INFO)
    assert info["converged"] == 1 and info["fell_back"] == 0
    assert info["rel_residual"] <= 1e-13 or info["backward_error"] <= 256 * 2.0 ** -53
    assert np.max(np.abs(got - want)) <= 1e-8 * np.max(np.abs(want))
