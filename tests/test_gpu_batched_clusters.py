"""GPU: systems of a batch that a thread-block cluster solves against the same systems on one CTA each.

The order of the operations on an entry depends neither on the panel width nor on who computes it, so the two agree
bit for bit: coefficients, values and reports.  Sizes around the cluster's 64-row tiles (n = 448 exactly, one row more,
a remainder of 1 to 63), the smallest and large ones, each alone (the cluster's share of a batch of one) and in a
batch that also has small systems for the single CTAs.
"""
import numpy as np
import pytest

import updes_gb300 as U
from functools import partial
from updes_gb300 import _lib
from updes_gb300.batched import LAST_BATCHED_INFO
from updes_gb300.rbf import gaussian, polyharmonic

pytestmark = pytest.mark.gpu

FACETS = {"North": "d", "South": "n", "West": "d", "East": "r"}


def _system(nx, ny, rbf, degree):
    cloud = U.SquareCloud(Nx=nx, Ny=ny, facet_types=dict(FACETS), jitter=(0.2, 3))
    g = lambda c: c[0] ** 2 - c[1]
    bcs = {f: (g, lambda c: 1.5 + 0.0 * c[0]) if k == "r" else g for f, k in FACETS.items()}
    return dict(diff_operator=lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial),
                rhs_operator=lambda x, centers, rbf, fields: np.sin(3 * x[0]) * np.cos(2 * x[1]), cloud=cloud,
                boundary_conditions=bcs, rbf=rbf, max_degree=degree)


def _solve(systems, precision, ctas):
    sols = U.pde_solver_batched(systems, precision=precision, tuner=None, ctas=ctas)
    return [(np.asarray(s.vals), np.asarray(s.coeffs)) for s in sols], [dict(i) for i in LAST_BATCHED_INFO]


def _same(systems, precision, alone):
    a, ia = _solve(systems, precision, 0)
    b, ib = _solve(systems, precision, 64)
    for k, (x, y) in enumerate(zip(a, b)):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]), (k, ia[k], ib[k])
        assert ia[k] == ib[k]
        assert np.all(np.isfinite(x[0]))
    if alone:
        assert ia[0]["lu_info"] == 0 and ia[0]["backward_error"] <= 1e-12


# (nx, ny, degree): n = nx ny + 1, 3 or 6 monomials.
SHAPES = [(21, 18, 2), (17, 26, 2), (18, 25, 0), (16, 27, 2), (23, 22, 2), (23, 25, 0), (31, 33, 0), (45, 45, 2)]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("shape", SHAPES)
def test_a_cluster_and_one_cta_agree(shape, precision):
    nx, ny, degree = shape
    _same([_system(nx, ny, partial(polyharmonic, a=1), degree)], precision, True)


def test_a_batch_for_clusters_and_single_ctas():
    systems = []
    for k, (nx, ny) in enumerate([(5, 6), (40, 41), (9, 7), (20, 21), (33, 30), (12, 12), (28, 17), (6, 5)] * 3):
        systems.append(_system(nx + k % 3, ny, partial(gaussian, eps=4.0) if k % 2 else partial(polyharmonic, a=1), 1))
    _same(systems, ["fp32" if k % 3 else "fp64" for k in range(len(systems))], False)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_a_singular_system_beside_a_regular_one(precision):
    """The zero operator without boundary columns leaves zero rows: the cluster reports the pivot that one CTA does, and
    the regular system keeps its bits."""
    good = _system(22, 22, partial(polyharmonic, a=1), 1)
    bad = _system(21, 23, partial(polyharmonic, a=1), 1)
    bad["diff_operator"] = lambda x, center, rbf, monomial, fields: 0.0 * U.nodal_laplacian(x, center, rbf, monomial)
    infos = []
    for ctas in (0, 64):
        with pytest.raises(_lib.UpdesError) as ei:
            U.pde_solver_batched([good, bad], precision=precision, tuner=None, ctas=ctas)
        assert ei.value.status == _lib.ERR_SINGULAR
        infos.append([dict(i) for i in LAST_BATCHED_INFO])
    assert infos[0][1]["lu_info"] == infos[1][1]["lu_info"] > 0
    assert infos[0][0] == infos[1][0] and infos[0][0]["lu_info"] == 0
