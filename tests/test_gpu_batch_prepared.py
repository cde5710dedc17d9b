"""GPU: prepared values (updes_eval_values_prepared) against a preparation that is not of the system given."""
import ctypes

import numpy as np
import pytest

import updes_gb300 as U
from updes_gb300 import _lib
from updes_gb300.multirhs import MultiRHSSolver

pytestmark = pytest.mark.gpu

FACETS = {"South": "d", "West": "d", "North": "d", "East": "d"}


def _op(x, center, rbf, monomial, fields=None):
    return U.nodal_value(x, center, rbf, monomial) - 0.01 * U.nodal_laplacian(x, center, rbf, monomial)


def _solver(nx, ny, degree, stretch=1.0, support_size="max"):
    ids = np.arange(nx * ny)
    coords = np.stack([np.linspace(0.0, stretch, nx)[ids // ny], np.linspace(0.0, 1.0, ny)[ids % ny]], axis=-1)
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=coords, facet_types=FACETS, support_size=support_size)
    return MultiRHSSolver(_op, cloud, {f: np.zeros(len(cloud.facet_nodes[f])) for f in FACETS}, U.polyharmonic, degree)


def _factor(dp, ws):
    co, info = U.SolverOptions(precision="fp64").c_opts(), _lib.SolveInfo()
    _lib.check(_lib.load().updes_factor(ctypes.byref(dp.c), ctypes.byref(co), ctypes.byref(info), ws.data_ptr(), ws.numel(),
                                        dp.stream()), "updes_factor")


def _values(dp, ws, bws):
    import torch
    lib = _lib.load()
    C = torch.ones((dp.n, 2), dtype=torch.float64, device="cuda")
    V = torch.zeros((dp.N, 2), dtype=torch.float64, device="cuda")
    _lib.check(lib.updes_eval_values_prepared(ctypes.byref(dp.c), 2, C.data_ptr(), 2, V.data_ptr(), 2, ws.data_ptr(),
                                              ws.numel(), bws.data_ptr(), bws.numel(), dp.stream()), "updes_eval_values_prepared")
    status = ctypes.c_int32(-1)
    _lib.check(lib.updes_workspace_status(ctypes.byref(dp.c), ws.data_ptr(), ws.numel(), ctypes.byref(status), dp.stream()),
               "updes_workspace_status")
    return V, status.value


def test_values_of_the_prepared_system():
    import torch
    s = _solver(9, 9, 1)
    V, status = _values(s.dp, s.ws, s.bws)
    assert torch.isfinite(V).all() and status == _lib.OK


@pytest.mark.parametrize("nx,ny,degree,refactor", [(9, 9, 1, True),      # another cloud of the same N and M
                                                   (13, 6, 2, True),     # the same n = 84, 78 + 6 instead of 81 + 3
                                                   (13, 6, 2, False)])
def test_a_preparation_of_another_system_gives_nan(nx, ny, degree, refactor):
    import torch
    s, other = _solver(9, 9, 1), _solver(nx, ny, degree, stretch=2.0)
    assert s.n == other.n
    if refactor:
        _factor(other.dp, s.ws)
    V, status = _values(other.dp, s.ws, s.bws)
    assert torch.isnan(V).all() and status == _lib.ERR_INVALID


def test_a_preparation_on_local_supports_has_no_values():
    import torch
    local, full = _solver(9, 9, 1, support_size=30), _solver(9, 9, 1)
    assert local.dp.c.support_width > 0 and full.dp.c.support_width == 0
    V, status = _values(full.dp, local.ws, local.bws)
    assert torch.isnan(V).all() and status == _lib.ERR_INVALID


@pytest.mark.parametrize("nx,ny,a,degree,substitution", [(30, 20, 1, 1, 1.2e-12), (40, 35, 2, 2, 8.0e-11), (24, 24, 3, 2, 5.2e-10)])
@pytest.mark.parametrize("R", [1, 9])
def test_triangles_are_solved_as_accurately_as_by_substitution(nx, ny, a, degree, substitution, R):
    # Values without a refinement sweep asked for, against the refined ones.  A substitution in 48-bit arithmetic leaves
    # 1.2e-12, 8e-11 and 5.2e-10 of the largest value (emulated on a CPU for r^3, r^5 and r^7); 32 times that.
    from functools import partial
    rng = np.random.default_rng(0)
    ids = np.arange(nx * ny)
    ii, jj = ids // ny, ids % ny
    coords = np.stack([np.linspace(0.0, 1.0, nx)[ii], np.linspace(0.0, 1.0, ny)[jj]], axis=-1)
    inner = (ii > 0) & (ii < nx - 1) & (jj > 0) & (jj < ny - 1)
    coords[inner] += rng.uniform(-0.2, 0.2, size=(nx * ny, 2))[inner] * min(1.0 / (nx - 1), 1.0 / (ny - 1))
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=coords, facet_types=FACETS)
    lap = lambda x, center, rbf, monomial, fields=None: U.nodal_laplacian(x, center, rbf, monomial)
    s = MultiRHSSolver(lap, cloud, {f: np.zeros(len(cloud.facet_nodes[f])) for f in FACETS},
                       partial(U.polyharmonic, a=a), degree, sweeps=0)
    x = np.asarray(cloud.sorted_nodes).T
    Q = np.stack([np.sin((3.0 + k) * x[0]) * np.cosh(x[1]) for k in range(R)], axis=1)
    plain = s.solve(Q)[1].cpu().numpy()
    s.sweeps = 4
    want = s.solve(Q)[1].cpu().numpy()
    assert np.max(np.abs(plain - want)) <= 32 * substitution * np.max(np.abs(want))
