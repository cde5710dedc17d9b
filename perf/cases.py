"""The work that users of this library have it do, as timed cases.

Each case is one call (or one short loop) through the public entry points:

* ``solve``: a fresh ``pde_solver`` call on host arrays, in either precision (no factors kept between calls);
* ``steps``: implicit time steps of R right-hand sides with ``MultiRHSSolver`` (factored once beforehand);
* ``grad``: ``pde_solver_torch`` and the gradient of a cost with respect to boundary control and fields;
* ``clouds``: many independent uneven clouds in one ``pde_solver_batched`` call;
* ``field``: value, gradient or Laplacian of a solved field at many points.

A solve returns the nodal solution.  The expansion coefficients are an intermediate of it that the collocation
systems (condition numbers up to 1e12) leave undetermined beyond about eight digits, so they are not compared;
the solution, the gradients and the fields are determined to 1e-10 and better on the systems used here, which
is why Neumann facets are left to the README example and the other kernels, why shape parameters scale with the
node spacing and why the control problem, whose gradient is a vector of such coefficients, has a Gaussian kernel.
"""
import math
from functools import partial

import numpy as np
import torch

import updes_gb300 as U
from updes_gb300.adjoint import pde_solver_torch
from updes_gb300.multirhs import MultiRHSSolver

FACETS = ("South", "West", "North", "East")
NORMAL = {"North": (0.0, 1.0), "South": (0.0, -1.0), "East": (1.0, 0.0), "West": (-1.0, 0.0)}
DT, KAPPA, VELOCITY = 1e-3, 0.01, (1.0, 0.5)


def listed():
    return [
        # the README example: Laplace on 30 x 20 uniform nodes, in the plain FP64 path and the default one.  The
        # smallest solves, where launches and host work count.
        _solve("readme_fp64", 30, 20, "nddd", "fp64", jitter=0.0, degree=1),
        _solve("readme_mixed", 30, 20, "nddd", "fp32", jitter=0.0, degree=1),
        # an everyday cloud of odd size with a variable coefficient and a Robin facet, default precision
        _solve("variable_mixed_61x47", 61, 47, "ddrd", "fp32", op="variable"),
        # the cloud of the boundary-control benchmark, default precision
        _solve("poisson_mixed_100x100", 100, 100, "dddd", "fp32"),
        # the headline Poisson system, the largest solve
        _solve("poisson_mixed_150x150", 150, 150, "dddd", "fp32"),
        # FP64 solves: a ragged mid-size cloud with a Gaussian kernel and a Neumann facet, and the largest one
        _solve("gaussian_fp64_67x59", 67, 59, "nddd", "fp64", rbf="gaussian", param=0.7),
        _solve("poisson_fp64_100x100", 100, 100, "dddd", "fp64"),
        # implicit advection-diffusion: 64 initial conditions at benchmark size, and a small ensemble
        dict(name="steps_80x80_r64", kind="steps", nx=80, ny=80, nrhs=64, steps=10),
        dict(name="steps_33x29_r7", kind="steps", nx=33, ny=29, nrhs=7, steps=30),
        # PDE-constrained control: cost and gradient, forward and reverse
        dict(name="control_gradient_50x50", kind="grad", nx=50, ny=50, precision="fp64"),
        # many uneven clouds at once
        dict(name="clouds_256", kind="clouds", count=256, low=10, high=45, shapes=0),
        # sampling the gradient of a solved field on a fine grid of points
        dict(name="field_gradient", kind="field", nx=100, ny=100, points=40000, what="gradient"),
    ]


def _solve(name, nx, ny, facets, precision, op="laplace", rbf="polyharmonic", param=1.0, degree=2, jitter=0.2):
    return dict(name=name, kind="solve", nx=nx, ny=ny, facets=facets, precision=precision, op=op, rbf=rbf,
                param=param, degree=degree, jitter=jitter)


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _sides(rng, low, high):
    """Nx, Ny of a cloud of about low..high nodes, up to twice as long one way as the other."""
    n, r = math.exp(rng.uniform(math.log(low), math.log(high))), math.exp(rng.uniform(-0.35, 0.35))
    nx = max(8, int(math.sqrt(n) * r))
    return nx, max(8, min(int(n / nx), int(high / nx)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "steps", "grad", "clouds", "field"])
    if kind == "solve":
        precision = rng.choice(["fp32", "fp64"])
        nx, ny = _sides(rng, 200, 22500 if precision == "fp32" else 10000)
        rbf, param, degree = rng.choice([("polyharmonic", 1.0, 1), ("polyharmonic", 1.0, 2), ("polyharmonic", 1.0, 2),
                                         ("gaussian", round(rng.uniform(0.6, 0.8), 3), 2),
                                         ("multiquadric", round(rng.uniform(0.8, 1.0), 3), 1)])
        if rbf != "polyharmonic":
            nx, ny = min(nx, 70), min(ny, 70)
        facets = rng.choice(["dddd", "dddd", "ddrd", "rddd"] if rbf == "polyharmonic" else ["dddd", "nddd", "ddrd"])
        return {k: v for k, v in _solve("", nx, ny, facets, precision, op=rng.choice(["laplace", "laplace", "variable"]),
                                        rbf=rbf, param=param, degree=degree).items() if k != "name"}
    if kind == "steps":
        nx, ny = _sides(rng, 400, 6400)
        return dict(kind="steps", nx=nx, ny=ny, nrhs=_log(rng, 1, 64), steps=_log(rng, 2, 30) if nx * ny < 2000 else
                    _log(rng, 2, 10))
    if kind == "grad":
        nx, ny = _sides(rng, 300, 3600)
        return dict(kind="grad", nx=nx, ny=ny, precision=rng.choice(["fp32", "fp64"]))
    if kind == "clouds":
        low = rng.randint(10, 20)
        return dict(kind="clouds", count=_log(rng, 8, 256), low=low, high=rng.randint(low + 5, 45),
                    shapes=rng.randint(1, 999))
    nx, ny = _sides(rng, 400, 10000)
    return dict(kind="field", nx=nx, ny=ny, points=_log(rng, 100, 40000), what=rng.choice(["value", "gradient",
                                                                                          "laplacian"]))


# ---- the grid, its node order and the data, made here from the seed ------------------------------------------

class _Grid:
    """Nodes of a jittered Nx x Ny grid by original id (i * Ny + j), and the solver's node order: interior,
    Dirichlet, Neumann, Robin, each by original id; corners belong to North, South, East, West in that order."""

    def __init__(self, nx, ny, facets, jitter, rng):
        self.nx, self.ny = nx, ny
        self.types = dict(zip(FACETS, facets))
        ids = np.arange(nx * ny)
        ii, jj = ids // ny, ids % ny
        self.coords = np.stack([np.linspace(0.0, 1.0, nx)[ii], np.linspace(0.0, 1.0, ny)[jj]], axis=-1)
        facet = np.where(jj == ny - 1, "North", np.where(jj == 0, "South", np.where(ii == nx - 1, "East", np.where(
            ii == 0, "West", ""))))
        h = min(1.0 / (nx - 1), 1.0 / (ny - 1))
        inner = facet == ""
        self.coords[inner] += rng.uniform(-jitter * h, jitter * h, size=(nx * ny, 2))[inner]
        kind = np.array([self.types.get(f, "i") for f in facet])
        order = np.concatenate([ids[kind == c] for c in "idnr"])
        self.X, self.facet, self.kind = self.coords[order], facet[order], kind[order]
        self.Ni = int(np.sum(self.kind == "i"))

    def cloud(self):
        return U.SquareCloud(Nx=self.nx, Ny=self.ny, coords=self.coords, facet_types=self.types)


class _Fourier:
    """A smooth random function on the unit square (vectorised over points) and its derivatives."""

    def __init__(self, rng, modes=8):
        self.a = rng.standard_normal(modes)
        self.k, self.l = rng.integers(1, 5, size=(2, modes))
        self.p, self.s = rng.uniform(0.0, 2.0, size=(2, modes))

    def __call__(self, x, dx=0, dy=0):
        d = lambda k, t, order: (np.pi * k) ** order * np.sin(np.pi * k * t + 0.5 * np.pi * order)
        return sum(a * d(k, x[0] + p, dx) * d(l, x[1] + s, dy)
                   for a, k, l, p, s in zip(self.a, self.k, self.l, self.p, self.s))


class _System:
    """The data of one solve, drawn from ``rng`` in a fixed order: the operator and boundary values of a smooth
    manufactured solution."""

    def __init__(self, case, rng):
        self.case = case
        self.grid = _Grid(case["nx"], case["ny"], case["facets"], case["jitter"], rng)
        self.u = _Fourier(rng)
        self.beta = float(rng.uniform(0.5, 2.0))
        amp = float(rng.uniform(0.3, 0.6))
        self.fields = _conductivity(self.grid.X.T, amp) if case["op"] == "variable" else None
        self.amp = amp
        self.param = case["param"]
        if case["rbf"] != "polyharmonic":  # shape parameters follow the node spacing
            self.param = _shape(case, self.param)

    def rhs(self, x):
        k, kx, ky = _conductivity(x, self.amp) if self.fields is not None else (1.0, 0.0, 0.0)
        return k * (self.u(x, 2, 0) + self.u(x, 0, 2)) + kx * self.u(x, 1, 0) + ky * self.u(x, 0, 1)

    def boundary(self, facet):
        x, (nx, ny) = self.grid.X[self.grid.facet == facet].T, NORMAL[facet]
        kind = self.grid.types[facet]
        value = 1.0 if kind == "d" else self.beta if kind == "r" else 0.0
        return value * self.u(x) + (0.0 if kind == "d" else nx * self.u(x, 1, 0) + ny * self.u(x, 0, 1))

    def arguments(self):
        grid = self.grid
        rbf = partial(getattr(U, self.case["rbf"]), **({"a": int(self.param)} if self.case["rbf"] == "polyharmonic"
                                                       else {"eps": self.param}))
        bcs = {}
        for name in FACETS:
            v = self.boundary(name)
            bcs[name] = (v, np.full(len(v), self.beta)) if grid.types[name] == "r" else v
        return dict(diff_operator=_div_k_grad if self.fields is not None else _laplacian,
                    rhs_operator=lambda x, centers, rbf, fields: self.rhs(x), cloud=grid.cloud(), boundary_conditions=bcs,
                    rbf=rbf, max_degree=self.case["degree"],
                    diff_args=None if self.fields is None else list(self.fields))

    def exact(self):
        grid = self.grid
        X = torch.as_tensor(grid.X, dtype=torch.float64, device=_device())
        W = torch.zeros((grid.Ni, 5), dtype=torch.float64, device=X.device)
        W[:, 3:] = 1.0
        if self.fields is not None:
            k, kx, ky = (torch.as_tensor(v[:grid.Ni], device=X.device) for v in self.fields)
            W = torch.stack([0.0 * k, kx, ky, k, k], dim=-1)
        K, A = _kansa(grid, X, W, self.case["rbf"], self.param, self.case["degree"], self.beta)
        q = np.zeros(K.shape[0])
        q[:grid.Ni] = self.rhs(grid.X[:grid.Ni].T)
        for name in FACETS:
            q[:len(grid.X)][grid.facet == name] = self.boundary(name)
        b = torch.as_tensor(q, device=X.device)
        return (A @ _solve_scaled(K, b)).cpu().numpy()


def _shape(case, shape):
    """A shape parameter in units of the node spacing."""
    return shape * (max(case["nx"], case["ny"]) - 1)


def _conductivity(x, amp):
    """k = 1 + amp sin(2 pi x) cos(2 pi y) and its derivatives."""
    s = 2.0 * np.pi
    return [1.0 + amp * np.sin(s * x[0]) * np.cos(s * x[1]), amp * s * np.cos(s * x[0]) * np.cos(s * x[1]),
            -amp * s * np.sin(s * x[0]) * np.sin(s * x[1])]


def _laplacian(x, center, rbf, monomial, fields):
    return U.nodal_laplacian(x, center, rbf, monomial)


def _div_k_grad(x, center, rbf, monomial, fields):
    g = U.nodal_gradient(x, center, rbf, monomial)
    return fields[0] * U.nodal_laplacian(x, center, rbf, monomial) + fields[1] * g[0] + fields[2] * g[1]


def _implicit_step(x, center, rbf, monomial, fields=None):
    g = U.nodal_gradient(x, center, rbf, monomial)
    return (U.nodal_value(x, center, rbf, monomial) / DT + VELOCITY[0] * g[0] + VELOCITY[1] * g[1]
            - KAPPA * U.nodal_laplacian(x, center, rbf, monomial))


def _bumps(grid, nrhs, rng):
    """Gaussian bumps (N, R), as the advection benchmark has them."""
    c, w = rng.uniform(0.3, 0.7, (nrhs, 2)), rng.uniform(0.05, 0.15, nrhs)
    d2 = (grid.X[:, None, 0] - c[None, :, 0]) ** 2 + (grid.X[:, None, 1] - c[None, :, 1]) ** 2
    return np.exp(-d2 / (2.0 * w[None, :] ** 2))


def _clouds(case, seed):
    shapes, rng = np.random.default_rng(case["shapes"]), np.random.default_rng(seed)  # the case's sizes, the seed's data
    systems = []
    for i in range(case["count"]):
        nx, ny = (int(v) for v in shapes.integers(case["low"], case["high"] + 1, size=2))
        rbf, param = [("gaussian", float(rng.uniform(0.6, 0.8))), ("polyharmonic", 1.0),
                      ("gaussian", float(rng.uniform(0.6, 0.8))), ("polyharmonic", 2.0 if nx * ny <= 900 else 1.0)][i % 4]
        facets = ("dddd", "rddd", "ddrd", "drdd")[int(shapes.integers(0, 4))]
        systems.append(_System(dict(nx=nx, ny=ny, facets=facets, op="laplace", rbf=rbf, param=param, degree=2,
                                    jitter=0.2), rng))
    return systems


def _control(case, seed):
    rng = np.random.default_rng(seed)
    grid = _Grid(case["nx"], case["ny"], "dddd", 0.2, rng)
    x = grid.X.T
    fields = _conductivity(x, float(rng.uniform(0.3, 0.6)))
    north = grid.X[grid.facet == "North"].T
    control = np.sin(np.pi * north[0]) * _Fourier(rng)(north)
    target = np.sinh(np.pi * x[1]) * np.sin(np.pi * x[0]) / np.sinh(np.pi)
    return grid, fields, control, target, _shape(case, 0.7)


def _field(case, seed):
    rng = np.random.default_rng(seed)
    grid = _Grid(case["nx"], case["ny"], "dddd", 0.2, rng)
    coeffs = np.concatenate([rng.standard_normal(len(grid.X)), rng.standard_normal(6)])
    return grid, coeffs, rng.uniform(0.0, 1.0, size=(case["points"], 2))


# ---- the interface -------------------------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "solve":
        options = U.SolverOptions(precision=case["precision"], reuse_factorization=False)
        return dict(kind=kind, call=dict(_System(case, rng).arguments(), options=options))
    if kind == "steps":
        grid = _Grid(case["nx"], case["ny"], "dddd", 0.0, rng)
        bcs = {f: np.zeros(int(np.sum(grid.facet == f))) for f in FACETS}
        solver = MultiRHSSolver(_implicit_step, grid.cloud(), bcs, partial(U.multiquadric, eps=_shape(case, 0.9)), 1)
        u0 = torch.as_tensor(_bumps(grid, case["nrhs"], rng), device="cuda")
        return dict(kind=kind, solver=solver, u0=u0, steps=case["steps"])
    if kind == "grad":
        grid, fields, control, target, eps = _control(case, seed)
        leaf = lambda v: torch.as_tensor(v, device="cuda").requires_grad_()
        zero = {f: np.zeros(int(np.sum(grid.facet == f))) for f in FACETS if f != "North"}
        return dict(kind=kind, cloud=grid.cloud(), zero=zero, fields=[leaf(v) for v in fields], control=leaf(control),
                    target=torch.as_tensor(target, device="cuda"), Ni=grid.Ni,
                    rbf=partial(U.gaussian, eps=eps), options=U.SolverOptions(precision=case["precision"]))
    if kind == "clouds":
        return dict(kind=kind, systems=[s.arguments() for s in _clouds(case, seed)])
    grid, coeffs, points = _field(case, seed)
    entry = {"value": U.value_vec, "gradient": U.gradient_vec, "laplacian": U.laplacian_vec}[case["what"]]
    return dict(kind=kind, entry=entry, points=points, coeffs=coeffs, centers=grid.X)


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return U.pde_solver(**state["call"]).vals
    if kind == "steps":
        return state["solver"].implicit_steps(state["u0"], state["steps"], 1.0 / DT)
    if kind == "grad":
        control, fields = state["control"], state["fields"]
        vals, _ = pde_solver_torch(_div_k_grad, lambda x, centers, rbf, fields: 0.0 * x[0], state["cloud"],
                                   dict(state["zero"], North=control), state["rbf"], 2, diff_args=fields,
                                   options=state["options"])
        cost = _cost(vals, state["target"], control, state["Ni"])
        return [cost.detach(), vals.detach(), *torch.autograd.grad(cost, [control, *fields])]
    if kind == "clouds":
        return np.concatenate([s.vals for s in U.pde_solver_batched(state["systems"])])
    return state["entry"](state["points"], state["coeffs"], state["centers"], U.polyharmonic)


def _cost(vals, target, control, Ni):
    return torch.mean((vals[:Ni] - target[:Ni]) ** 2) + 1e-4 * torch.sum(control ** 2)


def work(case):
    """Floating-point operations in the FP64 sense, and the bytes of inputs and outputs."""
    kind = case["kind"]
    if kind == "clouds":  # the mean of n^3 over the sizes that are drawn
        sides = range(case["low"], case["high"] + 1)
        m1, m3 = (sum(v ** p for v in sides) / len(sides) for p in (1, 3))
        return dict(flops=case["count"] * 2.0 / 3.0 * m3 * m3, bytes=case["count"] * m1 * m1 * 10 * 8.0)
    n = case["nx"] * case["ny"]
    if kind == "solve":
        return dict(flops=2.0 / 3.0 * n ** 3, bytes=10 * 8.0 * n)
    if kind == "grad":
        return dict(flops=2.0 / 3.0 * n ** 3 + 6.0 * n * n, bytes=20 * 8.0 * n)
    if kind == "steps":  # a forward and a backward triangle and the values, for each right-hand side; the factors once
        return dict(flops=case["steps"] * 4.0 * n * n * case["nrhs"],
                    bytes=case["steps"] * 8.0 * (n * n + 2.0 * n * case["nrhs"]))
    m = case["points"]
    return dict(flops=20.0 * m * n, bytes=8.0 * (3 * n + (4 if case["what"] == "gradient" else 3) * m))


# ---- the same results in plain 64-bit torch ------------------------------------------------------------------

def exact(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "solve":
        return _System(case, rng).exact()
    if kind == "clouds":
        return np.concatenate([s.exact() for s in _clouds(case, seed)])
    if kind == "steps":
        grid = _Grid(case["nx"], case["ny"], "dddd", 0.0, rng)
        u = torch.as_tensor(_bumps(grid, case["nrhs"], rng), device=_device())
        X = torch.as_tensor(grid.X, device=u.device)
        W = torch.tensor([1.0 / DT, *VELOCITY, -KAPPA, -KAPPA], dtype=torch.float64, device=u.device)
        K, A = _kansa(grid, X, W.expand(grid.Ni, 5), "multiquadric", _shape(case, 0.9), 1, 0.0)
        r, c = _scales(K)
        lu = torch.linalg.lu_factor(K * r[:, None] * c)
        for _ in range(case["steps"]):
            b = torch.zeros((K.shape[0], u.shape[1]), dtype=torch.float64, device=u.device)
            b[:grid.Ni] = u[:grid.Ni] / DT
            u = A @ (c[:, None] * torch.linalg.lu_solve(*lu, r[:, None] * b))
        return u
    if kind == "grad":
        return _exact_gradient(case, seed)
    grid, coeffs, points = _field(case, seed)
    X, c = (torch.as_tensor(v, device=_device()) for v in (grid.X, coeffs))
    out = []
    for p in torch.as_tensor(points, device=X.device).split(2048):
        t = [a @ c[:len(X)] for a in _kernel("polyharmonic", 1.0, p[:, None] - X[None])]
        t = [a + b @ c[len(X):] for a, b in zip(t, _monomials(2, p))]
        out.append({"value": t[0], "gradient": torch.stack(t[1:3], dim=-1), "laplacian": t[3] + t[4]}[case["what"]])
    return torch.cat(out).cpu().numpy()


def _exact_gradient(case, seed):
    grid, fields, control, target, eps = _control(case, seed)
    X = torch.as_tensor(grid.X, device=_device())
    k, kx, ky = (torch.as_tensor(v, device=X.device).requires_grad_() for v in fields)
    control = torch.as_tensor(control, device=X.device).requires_grad_()
    W = torch.stack([0.0 * k, kx, ky, k, k], dim=-1)[:grid.Ni]
    K, A = _kansa(grid, X, W, "gaussian", eps, 2, 0.0)
    north = torch.as_tensor(np.flatnonzero(grid.facet == "North"), device=X.device)
    b = torch.zeros(K.shape[0], dtype=torch.float64, device=X.device).index_put((north,), control)
    vals = A @ _solve_scaled(K, b)
    cost = _cost(vals, torch.as_tensor(target, device=X.device), control, grid.Ni)
    return [cost.detach(), vals.detach(), *torch.autograd.grad(cost, [control, k, kx, ky])]


def _scales(K):
    """Powers of two that bring the rows and then the columns of K to about 1."""
    r = 2.0 ** -torch.round(torch.log2(K.detach().abs().amax(1)))
    return r, 2.0 ** -torch.round(torch.log2((K.detach() * r[:, None]).abs().amax(0)))


def _solve_scaled(K, b):
    r, c = _scales(K)
    return c * torch.linalg.solve(K * r[:, None] * c, b * r)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _kernel(rbf, param, d):
    """Value, gradient and the two second derivatives of the kernel at the differences d (..., 2); derivatives are
    0 at d = 0."""
    dx, dy = d[..., 0], d[..., 1]
    r2 = dx * dx + dy * dy
    if rbf == "polyharmonic":
        p = 2 * int(param) + 1
        r = r2.sqrt()
        phi, g1 = r ** p, p * r ** (p - 2)
        g2 = torch.where(r2 > 0, p * (p - 2) * torch.where(r2 > 0, r, 1.0) ** (p - 4), 0.0)
    elif rbf == "gaussian":
        phi = torch.exp(-param * param * r2)
        g1, g2 = -2.0 * param ** 2 * phi, 4.0 * param ** 4 * phi
    else:
        phi = torch.sqrt(1.0 + param * param * r2)
        g1, g2 = param ** 2 / phi, -param ** 4 / phi ** 3
    some = r2 > 0
    return phi, g1 * dx, g1 * dy, torch.where(some, g1 + g2 * dx * dx, 0.0), torch.where(some, g1 + g2 * dy * dy, 0.0)


def _monomials(degree, X):
    """The same five terms of x^a y^b, a + b <= degree, by total degree and then falling a; each (m, M)."""
    x, y = X[:, 0], X[:, 1]
    power = lambda v, e: v ** e if e >= 0 else 0.0 * v
    exps = [(t - b, b) for t in range(degree + 1) for b in range(t + 1)]
    terms = [lambda a, b: power(x, a) * power(y, b), lambda a, b: a * power(x, a - 1) * power(y, b),
             lambda a, b: b * power(x, a) * power(y, b - 1),
             lambda a, b: a * (a - 1) * power(x, a - 2) * power(y, b),
             lambda a, b: b * (b - 1) * power(x, a) * power(y, b - 2)]
    return [torch.stack([f(a, b) for a, b in exps], dim=-1) for f in terms]


def _kansa(grid, X, W, rbf, param, degree, beta):
    """K = [[op Phi, op P], [bd Phi, bd P], [P^T, 0]] and A = [Phi P], the diagonal of the Phi blocks zero."""
    N, Ni = len(grid.X), grid.Ni
    t, m = _kernel(rbf, param, X[:, None] - X[None]), _monomials(degree, X)
    P = m[0]
    full = lambda a, b: torch.cat([a, b], dim=1)
    off = 1.0 - torch.eye(N, dtype=torch.float64, device=X.device)
    A = full(t[0] * off, P)
    top = sum(W[:, i:i + 1] * full(t[i][:Ni], m[i][:Ni]) for i in range(5))
    nx, ny, robin, slope = (torch.as_tensor(v[Ni:, None], device=X.device) for v in (
        np.array([NORMAL.get(f, (0.0, 0.0))[0] for f in grid.facet]),
        np.array([NORMAL.get(f, (0.0, 0.0))[1] for f in grid.facet]),
        np.where(grid.kind == "d", 1.0, np.where(grid.kind == "r", beta, 0.0)),
        np.where(grid.kind == "d", 0.0, 1.0)))
    v, gx, gy = (full(t[i][Ni:], m[i][Ni:]) for i in range(3))
    bottom = robin * v + slope * (nx * gx + ny * gy)
    body = torch.cat([top, bottom]) * full(off, torch.ones_like(P))
    last = full(P.T, torch.zeros((P.shape[1], P.shape[1]), dtype=torch.float64, device=X.device))
    return torch.cat([body, last]), A
