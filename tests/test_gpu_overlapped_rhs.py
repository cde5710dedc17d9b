"""GPU: the right-hand side of a fresh solve is formed while the GPU factors (updes_solve_begin / updes_solve_end).

The result is updes_solve's bit for bit, whatever the right-hand side does meanwhile: solve another system, evaluate a field,
fail; the workspace is back in the cache afterwards and the next solve is not disturbed.
"""
from functools import partial

import numpy as np
import pytest

import updes_gb300 as U
from updes_gb300 import operators as O

pytestmark = pytest.mark.gpu


def _lap(x, center, rbf, monomial, fields):
    return U.nodal_laplacian(x, center, rbf, monomial)


def _args(nx, ny, rhs):
    cloud = U.SquareCloud(Nx=nx, Ny=ny, facet_types={"North": "d", "South": "n", "West": "d", "East": "d"})
    bcs = {f: (lambda c: c[0] - c[1]) for f in ("North", "South", "West", "East")}
    return dict(diff_operator=_lap, rhs_operator=rhs, cloud=cloud,
                boundary_conditions=O.boundary_conditions_func_to_arr(bcs, cloud),
                rbf=partial(U.polyharmonic, a=1), max_degree=1)


def _plain(x, centers, rbf, fields):
    return np.sin(3 * x[0]) * x[1]


def _separate(a, options):
    """The same solve from the whole preparation and one updes_solve."""
    W, kind, bn, geom, q = O.prepare(a["diff_operator"], a["rhs_operator"], a["cloud"], a["boundary_conditions"],
                                     a["rbf"], a["max_degree"], options=options)
    dp = O.DeviceProblem(a["cloud"], a["rbf"], a["max_degree"], W, kind, bn, geom)
    c, v, _ = O.solve_device(dp, q, options)
    return c.cpu().numpy(), v.cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(4, 4), (17, 15), (40, 33)])
def test_same_as_one_call(shape, precision):
    options = U.SolverOptions(precision=precision, reuse_factorization=False)
    a = _args(*shape, _plain)
    want = _separate(a, options)
    got = U.pde_solver(**a, options=options)
    assert np.array_equal(got.coeffs, want[0]) and np.array_equal(got.vals, want[1])


def test_a_right_hand_side_that_solves():
    options = U.SolverOptions(precision="fp32", reuse_factorization=False)
    inner = _args(20, 19, _plain)
    seen = []

    def rhs(x, centers, rbf, fields):
        seen.append(U.pde_solver(**inner, options=options).vals)
        return _plain(x, centers, rbf, fields)
    a = _args(35, 31, _plain)
    want, want_inner = _separate(a, options), _separate(inner, options)
    got = U.pde_solver(**dict(a, rhs_operator=rhs), options=options)
    assert np.array_equal(got.vals, want[1]) and np.array_equal(seen[0], want_inner[1])


def test_a_right_hand_side_that_fails():
    options = U.SolverOptions(precision="fp64", reuse_factorization=False)
    a = _args(20, 19, _plain)
    want = _separate(a, options)

    def fails(x, centers, rbf, fields):
        raise KeyError("rhs")
    for bad in (fails, lambda x, centers, rbf, fields: np.nan):
        with pytest.raises((KeyError, ValueError)):
            U.pde_solver(**dict(a, rhs_operator=bad), options=options)
        assert np.array_equal(U.pde_solver(**a, options=options).vals, want[1])
    assert len(O._WS_CACHE) == 1


def _batch(count):
    """Systems of 16 to 72 nodes, every 9th of 600 (for the clusters), the kernels alternating."""
    out = []
    for k in range(count):
        a = _args(*((4 + k % 5, 4 + k % 6) if k % 9 else (25, 24)), _plain)
        if k % 2:
            a["rbf"] = partial(U.gaussian, eps=4.0)
        out.append(a)
    return out


@pytest.mark.parametrize("precision", ["fp64", "auto"])
def test_a_batch_in_parts(precision):
    """A batch that is prepared and launched in parts gives what its pieces of one part each give."""
    from updes_gb300.batched import LAST_BATCHED_INFO, _parts
    systems = _batch(150)
    assert len(_parts([s["cloud"].N for s in systems])) > 2
    got = U.pde_solver_batched(systems, precision=precision, tuner=None)
    infos = [dict(i) for i in LAST_BATCHED_INFO]
    for first in (0, 50, 100):
        want = U.pde_solver_batched(systems[first:first + 50], precision=precision, tuner=None)
        assert infos[first:first + 50] == [dict(i) for i in LAST_BATCHED_INFO]
        for g, w in zip(got[first:first + 50], want):
            assert np.array_equal(g.vals, w.vals) and np.array_equal(g.coeffs, w.coeffs)


def test_a_batch_whose_last_part_fails():
    systems = _batch(150)

    def fails(x, centers, rbf, fields):
        raise KeyError("rhs")
    with pytest.raises(KeyError):
        U.pde_solver_batched(systems[:-1] + [dict(systems[-1], rhs_operator=fails)], precision="fp64", tuner=None)
    a, b = (U.pde_solver_batched(systems[:20], precision="fp64", tuner=None) for _ in range(2))
    assert all(np.array_equal(x.vals, y.vals) for x, y in zip(a, b))
