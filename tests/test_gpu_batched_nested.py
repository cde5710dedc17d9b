"""GPU: a caller's function that solves a batch of its own, on another stream, while parts of the batch run."""
from functools import partial

import numpy as np
import pytest

import updes_gb300 as U

pytestmark = pytest.mark.gpu


def _lap(x, center, rbf, monomial, fields):
    return U.nodal_laplacian(x, center, rbf, monomial)


def _plain(x, centers, rbf, fields):
    return np.sin(3 * x[0]) * x[1]


def _system(nx, ny, rhs=_plain):
    return dict(diff_operator=_lap, rhs_operator=rhs, cloud=U.SquareCloud(Nx=nx, Ny=ny, facet_types=dict.fromkeys(
                    ("North", "South", "West", "East"), "d")),
                boundary_conditions={f: (lambda c: c[0] - c[1]) for f in ("North", "South", "West", "East")},
                rbf=partial(U.polyharmonic, a=1), max_degree=1)


def test_a_batch_inside_a_batch():
    import torch
    inner = [_system(20 + k % 3, 21) for k in range(12)]
    sizes = [(18 + k % 7, 20) for k in range(150)]
    solve = lambda systems: [s.vals for s in U.pde_solver_batched(systems, precision="fp64", tuner=None)]
    want, want_inner = solve([_system(*s) for s in sizes]), solve(inner)
    seen = []

    def rhs(x, centers, rbf, fields):
        with torch.cuda.stream(torch.cuda.Stream()):
            seen.append(solve(inner))
        return _plain(x, centers, rbf, fields)
    got = solve([_system(*s, rhs=rhs if k in (60, 149) else _plain) for k, s in enumerate(sizes)])
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert len(seen) == 2 and all(np.array_equal(a, b) for s in seen for a, b in zip(s, want_inner))
