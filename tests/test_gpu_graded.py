"""GPU: the FP64 paths on matrices whose rows and columns are of very different size.  A collocation matrix of r^(2a+1) on
a domain of side S has kernel entries of S^(2a+1) beside the ones of its polynomial block."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nodes(nx, ny, side, seed=None):
    rng = np.random.default_rng(nx * ny if seed is None else seed)
    ids = np.arange(nx * ny)
    ii, jj = ids // ny, ids % ny
    X = np.stack([np.linspace(0.0, 1.0, nx)[ii], np.linspace(0.0, 1.0, ny)[jj]], axis=-1)
    inner = (ii > 0) & (ii < nx - 1) & (jj > 0) & (jj < ny - 1)
    X[inner] += rng.uniform(-0.2, 0.2, size=(nx * ny, 2))[inner] * min(1.0 / (nx - 1), 1.0 / (ny - 1))
    return X * side


def _lu(A):
    import torch
    from updes_gb300 import _lib
    lib = _lib.load()
    n = A.shape[0]
    ld = int(lib.updes_matrix_ld(n, 8))
    F = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    F[:, :n] = torch.as_tensor(A)
    piv = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    nb, info = ctypes.c_size_t(), ctypes.c_int32(-1)
    _lib.check(lib.updes_lu_workspace(n, _lib.PREC_FP64, ctypes.byref(nb)), "updes_lu_workspace")
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    _lib.check(lib.updes_lu_factor(n, F.data_ptr(), ld, _lib.PREC_FP64, F.data_ptr(), ld, piv.data_ptr(), ws.data_ptr(),
                                   ws.numel(), ctypes.byref(info),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "updes_lu_factor")
    assert info.value == 0
    LU, PA = F.cpu().numpy()[:, :n], A[piv.cpu().numpy()[n:]]
    return PA, np.tril(LU, -1) + np.eye(n), np.triu(LU)


def _graded(kind, n):
    if kind == "rows":
        rng = np.random.default_rng(n)
        return rng.standard_normal((n, n)) * 2.0 ** rng.integers(-60, 60, (n, 1))
    nx, ny = (n - 3) // 20, 20
    X = _nodes(nx, ny, 2.0 ** -10)
    r = np.sqrt(((X[:, None] - X[None]) ** 2).sum(-1))
    P = np.concatenate([np.ones((len(X), 1)), X], axis=1)
    return np.block([[r ** (3 if kind == "r3" else 5), P], [P.T, np.zeros((3, 3))]])


@pytest.mark.parametrize("kind,n", [("rows", 33), ("rows", 300), ("rows", 1100), ("r3", 603), ("r5", 403), ("r3", 1203)])
def test_lu_factor_takes_any_scaling(kind, n):
    # a chain of multiply-adds per entry: |PA - LU| <= n u |L||U|, and the check's own product once more
    A = _graded(kind, n)
    PA, L, U = _lu(A)
    wrong = np.abs(PA - L @ U) > 2 * A.shape[0] * 2.0 ** -53 * (np.abs(L) @ np.abs(U))
    assert not wrong.any(), f"{int(wrong.sum())} entries"


def _poisson(side, a, precision, nx=30, ny=20, degree=2):
    import updes_gb300 as U
    from functools import partial
    X = _nodes(nx, ny, side)
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=X, facet_types={f: "d" for f in ("South", "West", "North", "East")})
    x = np.asarray(cloud.sorted_nodes).T / side
    values = np.sin(x[0]) * np.exp(x[1])
    bcs = {f: values[np.asarray(cloud.facet_nodes[f])] for f in cloud.facet_types}
    rhs = lambda x, centers, rbf, fields: np.sin(3.0 * x[0] / side) * np.cosh(2.0 * x[1] / side) / side ** 2
    lap = lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial)
    return U.pde_solver(lap, rhs, cloud, bcs, partial(U.polyharmonic, a=a), degree,
                        options=U.SolverOptions(precision=precision, reuse_factorization=False))


# A domain whose side is a power of two is the unit square's system with exactly scaled coordinates and entries, so the
# nodal values are those of side 1 up to the errors of an FP64 solution on it.  LAPACK's (CPU, against extended precision,
# four clouds): 8e-14 for r^3 and 2.3e-12 for r^5; 32 times that for the two solutions compared.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("a,degree,lapack", [(1, 1, 8e-14), (1, 2, 8e-14), (2, 2, 2.3e-12)])
@pytest.mark.parametrize("k", [-13, -10, -7, 4])
def test_the_solution_does_not_depend_on_the_unit_of_length(k, a, degree, lapack, precision):
    from updes_gb300 import operators
    want = _poisson(1.0, a, "fp64", degree=degree).vals
    got = _poisson(2.0 ** k, a, precision, degree=degree).vals
    # a mixed solve that its refinement certifies (256 u of backward error) is held to that
    certified = precision == "fp32" and not operators.LAST_INFO["fell_back"]
    assert np.max(np.abs(got - want)) <= (256 if certified else 1) * 32 * lapack * np.max(np.abs(want))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_the_adjoint_on_a_small_domain(precision):
    # A cost w . vals is linear in the boundary values, so its gradient times other boundary values is the cost of their
    # solution.  The gradient itself is a vector of coefficients, which r^3 leaves undetermined beyond eight digits; a
    # transposed solution of small backward error gives the product as well as a solution gives its values.
    import torch
    import updes_gb300 as U
    from functools import partial
    from updes_gb300.adjoint import pde_solver_torch
    lap = lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial)
    w = np.random.default_rng(1).standard_normal(600)

    def solve(side, precision, value):
        cloud = U.SquareCloud(Nx=30, Ny=20, coords=_nodes(30, 20, side),
                              facet_types={f: "d" for f in ("South", "West", "North", "East")})
        x = np.asarray(cloud.sorted_nodes).T / side
        bcs = {f: np.zeros(len(cloud.facet_nodes[f])) for f in cloud.facet_types}
        control = torch.as_tensor(value(x[0][np.asarray(cloud.facet_nodes["North"])]), device="cuda").requires_grad_()
        vals, _ = pde_solver_torch(lap, lambda x, centers, rbf, fields: 0.0 * x[0], cloud, dict(bcs, North=control),
                                   partial(U.polyharmonic, a=1), 1, options=U.SolverOptions(precision=precision))
        return control, vals

    other = lambda t: np.cos(2.0 * t)
    control, vals = solve(2.0 ** -10, precision, lambda t: np.sin(np.pi * t))  # fp32 falls back to FP64 on this side
    gradient, = torch.autograd.grad(torch.dot(torch.as_tensor(w, device="cuda"), vals), [control])
    control, vals = solve(1.0, "fp64", other)
    vals = vals.detach().cpu().numpy()
    got = float(torch.dot(gradient, control.detach()))
    assert abs(got - w @ vals) <= 64 * 8e-14 * np.abs(w).sum() * np.max(np.abs(vals))


def test_far_nodes_do_not_spoil_the_scaling():
    # a facet whose nodes see the others' Gaussians at 1e-10 only: their rows are all polynomial, and its values come out
    # as those of the polynomial that the data are (FP64 arithmetic on a CPU: 2.6e-12)
    import updes_gb300 as U
    from functools import partial
    nx, ny = 20, 16
    ii, jj = np.arange(nx * ny) // ny, np.arange(nx * ny) % ny
    X = np.stack([np.linspace(0.0, 1.0, nx)[ii], np.linspace(0.0, 1.0, ny)[jj]], axis=-1)
    X[ii == nx - 1] = np.stack([np.full(ny, 1.4), 6.0 * np.linspace(0.0, 1.0, ny)], axis=-1)
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=X, facet_types={f: "d" for f in ("South", "West", "North", "East")})
    x = np.asarray(cloud.sorted_nodes).T
    exact = 1.0 + 0.3 * x[0] - 0.2 * x[1]
    bcs = {f: exact[np.asarray(cloud.facet_nodes[f])] for f in cloud.facet_types}
    lap = lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial)
    sol = U.pde_solver(lap, lambda x, centers, rbf, fields: 0.0 * x[0], cloud, bcs, partial(U.gaussian, eps=12.0), 1,
                       options=U.SolverOptions(precision="fp64", reuse_factorization=False))
    assert np.max(np.abs(sol.vals - exact)) <= 3e-10


@pytest.mark.parametrize("squeeze", [(0.001, 1.0), (0.01, 0.01)])
def test_kernels_that_decouple_most_nodes(squeeze):
    # Gaussians scaled to the finest spacing of an anisotropic (or half squeezed) cloud: K stays graded whatever its scaling,
    # and the solution has to come out as FP64 multiply-adds give it.  LAPACK's lies within 2e-13 and 1e-11 of extended
    # precision (four clouds each); 16 times what it gives here, and never less than 16 times 2e-14.
    import scipy.linalg as sl
    import updes_gb300 as U
    from functools import partial
    nx, ny, wide = 36, 24, np.longdouble
    X = _nodes(nx, ny, 1.0, seed=0)
    X = X * squeeze if squeeze[1] == 1.0 else np.where(X[:, :1] < 0.5, X * squeeze, X)
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=X, facet_types={f: "d" for f in ("South", "West", "North", "East")})
    X = np.asarray(cloud.sorted_nodes)
    N, Ni = cloud.N, cloud.Ni
    d2 = ((X[:, None] - X[None]) ** 2).sum(-1)
    eps = 0.8 / np.median(np.sqrt((d2 + 9.0 * np.eye(N)).min(1)))
    low, span = X.min(0), X.max(0) - X.min(0)
    x = ((X - low) / span).T
    values = np.sin(2.0 * x[0]) * np.exp(x[1])
    bcs = {f: values[np.asarray(cloud.facet_nodes[f])] for f in cloud.facet_types}
    lap = lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial)
    rhs = lambda x: np.cos(3.0 * (x[0] - low[0]) / span[0] + (x[1] - low[1]) / span[1]) / np.max(span) ** 2
    got = U.pde_solver(lap, lambda x, centers, rbf, fields: rhs(x), cloud, bcs, partial(U.gaussian, eps=eps), 1,
                       options=U.SolverOptions(precision="fp64", reuse_factorization=False)).vals
    # the same system in extended precision: K c = q with the kernels' own diagonal left out, A c at the nodes
    Xw, e2 = X.astype(wide), wide(eps) ** 2
    r2 = (Xw[:, None, 0] - Xw[None, :, 0]) ** 2 + (Xw[:, None, 1] - Xw[None, :, 1]) ** 2
    phi = np.exp(-e2 * r2)
    np.fill_diagonal(phi, 0.0)
    P = np.concatenate([np.ones((N, 1), wide), Xw], axis=1)
    A = np.concatenate([phi, P], axis=1)
    K = np.concatenate([A, np.concatenate([P.T, np.zeros((3, 3), wide)], axis=1)])
    K[:Ni, :N] = ((4.0 * e2 * e2 * r2 - 4.0 * e2) * phi)[:Ni]
    K[:Ni, N:] = 0.0
    q = np.concatenate([rhs(X[:Ni].T), values[Ni:], np.zeros(3)])
    size = lambda m: 2.0 ** -np.frexp(m.astype(float))[1].astype(float)
    r = size(np.abs(K).max(1))
    c = size(np.abs(K * r[:, None]).max(0))
    lu = sl.lu_factor((K * r[:, None] * c).astype(float))
    y = sl.lu_solve(lu, r * q)
    lapack = (A @ (c * y)).astype(float)
    y = y.astype(wide)
    for _ in range(4):
        y = y + sl.lu_solve(lu, (r * (q - K @ (c * y))).astype(float))
    want = (A @ (c * y)).astype(float)
    error = lambda v: np.max(np.abs(v - want)) / np.max(np.abs(want))
    assert error(got) <= 16.0 * max(error(lapack), 2e-14)


@pytest.mark.parametrize("side", [1.0, 2.0 ** -7, 2.0 ** -10])
@pytest.mark.parametrize("nx,ny,a,degree", [(30, 20, 1, 1), (16, 16, 1, 2), (40, 13, 2, 2)])
def test_time_step_values_on_a_small_domain(side, nx, ny, a, degree):
    # vals = Phi C + P C: the kernel part from digits cut at 2^-56 of the largest entry of a row (column) in a block of 256
    # columns (rows), twice 256 cuts of at most 2^-55 with the products left out; the sums and the polynomial part in FP64
    import updes_gb300 as U
    from functools import partial
    from updes_gb300.multirhs import MultiRHSSolver
    op = lambda x, center, rbf, monomial, fields=None: (U.nodal_value(x, center, rbf, monomial)
                                                        - 0.01 * side ** 2 * U.nodal_laplacian(x, center, rbf, monomial))
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=_nodes(nx, ny, side),
                          facet_types={f: "d" for f in ("South", "West", "North", "East")})
    s = MultiRHSSolver(op, cloud, {f: np.zeros(len(cloud.facet_nodes[f])) for f in cloud.facet_types},
                       partial(U.polyharmonic, a=a), degree)
    X = np.asarray(cloud.sorted_nodes)
    x = X.T / side
    C, V = (t.cpu().numpy() for t in s.solve(np.stack([np.sin(3.0 * x[0]) * np.exp(x[1]), np.cos(x[0] + 2.0 * x[1])], axis=1)))
    wide = np.longdouble
    Xw = X.astype(wide)
    phi = np.sqrt((Xw[:, None, 0] - Xw[None, :, 0]) ** 2 + (Xw[:, None, 1] - Xw[None, :, 1]) ** 2) ** (2 * a + 1)
    powers = [(i - j, j) for i in range(degree + 1) for j in range(i + 1)]
    P = np.stack([Xw[:, 0] ** i * Xw[:, 1] ** j for i, j in powers], axis=-1)
    N = len(X)
    want = (phi @ C[:N] + P @ C[N:]).astype(float)
    bound = 16 * 2.0 ** -53 * (np.abs(phi) @ np.abs(C[:N]) + np.abs(P) @ np.abs(C[N:])).astype(float)
    for k in range(0, N, 256):
        bound += 512 * 2.0 ** -55 * np.outer(np.abs(phi[:, k:k + 256]).max(1), np.abs(C[k:min(k + 256, N)]).max(0)).astype(float)
    wrong = np.abs(V - want) > bound
    assert not wrong.any(), f"{int(wrong.sum())} values, by up to {np.max(np.abs(V - want) / bound):.1e} of the bound"


@pytest.mark.parametrize("index", [12, 24, 36])
def test_flat_kernels_are_not_factored_again(index):
    # a Gaussian that is singular to working precision: a large backward error (FP64 multiply-adds: 1e-10 as well) that no
    # factors can lower, so as many panels as r^3 takes on the same cloud
    from functools import partial
    import updes_gb300 as U
    from updes_gb300 import _lib, operators, workloads
    system = workloads.uneven_clouds(index + 1)[index]

    def panels(rbf):
        _lib.stats_reset(timing=True)
        U.pde_solver(**dict(system, rbf=rbf), options=U.SolverOptions(precision="fp64", reuse_factorization=False))
        count = _lib.stats_read()["by_class"]["panel"]["count"]
        _lib.stats_reset()
        return count, operators.LAST_INFO["backward_error"]

    (once, small), (count, large) = panels(partial(U.polyharmonic, a=1)), panels(system["rbf"])
    assert small < 2.0 ** -46 and large > 2.0 ** -40
    assert count == once > 0


def test_quintic_kernel_on_two_spacings():
    # r^5 with half of the nodes at 0.03 of the others' spacing, a backward error hardly above the usual: the values as FP64
    # multiply-adds give them.  LAPACK's lie 1.2e-7 from extended precision; 16 times what it gives here.
    import scipy.linalg as sl
    import updes_gb300 as U
    from functools import partial
    nx, ny, wide = 22, 16, np.longdouble
    X = _nodes(nx, ny, 1.0, seed=0)
    X = np.where(X[:, :1] < 0.5, X * 0.03, X)
    cloud = U.SquareCloud(Nx=nx, Ny=ny, coords=X, facet_types={f: "d" for f in ("South", "West", "North", "East")})
    X = np.asarray(cloud.sorted_nodes)
    N, Ni = cloud.N, cloud.Ni
    low, span = X.min(0), X.max(0) - X.min(0)
    x = ((X - low) / span).T
    values = np.sin(2.0 * x[0]) * np.exp(x[1])
    bcs = {f: values[np.asarray(cloud.facet_nodes[f])] for f in cloud.facet_types}
    lap = lambda x, center, rbf, monomial, fields: U.nodal_laplacian(x, center, rbf, monomial)
    rhs = lambda x: np.cos(3.0 * (x[0] - low[0]) / span[0] + (x[1] - low[1]) / span[1]) / np.max(span) ** 2
    got = U.pde_solver(lap, lambda x, centers, rbf, fields: rhs(x), cloud, bcs, partial(U.polyharmonic, a=2), 2,
                       options=U.SolverOptions(precision="fp64", reuse_factorization=False)).vals
    Xw = X.astype(wide)
    r2 = ((Xw[:, None] - Xw[None]) ** 2).sum(-1)
    x, y = Xw.T
    P = np.stack([np.ones(N, wide), x, y, x * x, x * y, y * y], axis=1)
    A = np.concatenate([np.sqrt(r2) * r2 * r2, P], axis=1)
    K = np.concatenate([A, np.concatenate([P.T, np.zeros((6, 6), wide)], axis=1)])
    K[:Ni, :N] = (25.0 * np.sqrt(r2) * r2)[:Ni]
    K[:Ni, N:] = np.array([0, 0, 0, 2, 0, 2], wide)
    q = np.concatenate([rhs(X[:Ni].T), values[Ni:], np.zeros(6)])
    size = lambda m: 2.0 ** -np.frexp(m.astype(float))[1].astype(float)
    r = size(np.abs(K).max(1))
    c = size(np.abs(K * r[:, None]).max(0))
    lu = sl.lu_factor((K * r[:, None] * c).astype(float))
    y = sl.lu_solve(lu, r * q)
    lapack = (A @ (c * y)).astype(float)
    y = y.astype(wide)
    for _ in range(8):
        y = y + sl.lu_solve(lu, (r * (q - K @ (c * y))).astype(float))
    want = (A @ (c * y)).astype(float)
    error = lambda v: np.max(np.abs(v - want)) / np.max(np.abs(want))
    assert error(got) <= 16.0 * error(lapack)
