"""The work that programs have this framework do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` builds what a user's program holds before the
call (the problem, the solver with its assembled matrix and preconditioner, the state reached
so far), ``run`` is one pass through the public entry points, ``work`` the bytes and flops that
a pass cannot do without and ``exact`` the same outputs from dense or element-wise FP64 algebra
without this package's code (where that is affordable).

Calls:
  loop      one pass of the ``solve_direct`` time loop (right-hand side and solve)
  step      ``MPETSolver.step``: assembly, right-hand side, solve
  batch     one loop pass of ``MPETBatchSolver`` over many instances
  adjoint   ``pressure_misfit`` and its backward pass with respect to per-cell K
  estimate  ``AdaptiveMPETSolver.indicators``
  operator  ``mpet_assemble``, ``mpet_rhs``, ``mpet_residual`` and ``mpet_spmv`` of the C ABI
"""
import gc
import math

import numpy as np
import torch

from waterscapes_gb300 import (AdaptiveMPETSolver, CompiledSubDomain, Constant, EllipsoidShellMesh, Expression,
                               MPETBatchSolver, MPETProblem, MPETSolver, MPETTotalPressureSolver, UnitCubeMesh,
                               UnitSquareMesh, convert_to_E_nu)
from waterscapes_gb300 import _lib
from waterscapes_gb300.adjoint import pressure_misfit

MESHES = {"cube": UnitCubeMesh, "square": UnitSquareMesh, "shell": EllipsoidShellMesh}
DIRICHLET, NEUMANN, ROBIN = 0, 1, 2


def _case(name, **kw):
    c = {"call": "loop", "mesh": "cube", "n": 8, "J": 2, "precision": "mixed", "theta": 1.0, "form": "mpet",
         "boundary": "dirichlet", "K": "constant", "S": "symmetric", "rtol": 1e-11}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a unit-test sized problem: many small launches, latency only
        _case("cube 4, A=2", n=4),
        # the plain FP64 workload: A=2 on 16^3, backward Euler
        _case("cube 16, A=2, fp64", n=16, precision="fp64"),
        # FP64 end to end with four networks
        _case("cube 28, A=4, fp64", n=28, J=4, precision="fp64"),
        # an odd size with traction, flux and Robin boundaries and sources, the matrix assembled
        # in every step (MPETSolver.step), Crank-Nicolson
        _case("cube 21, A=2, step", call="step", n=21, theta=0.5, boundary="mixed"),
        # the headline workload: 64^3, four networks, mixed precision, rtol of that workload
        _case("cube 64, A=4", n=64, J=4, rtol=1e-10),
        # an unstructured, jittered shell with a log-normal permeability per cell
        _case("shell 11, A=4, K per cell", mesh="shell", n=11, J=4, K="cells"),
        # the reference's own 2D rate tests: non-symmetric transfer, hence GMRES
        _case("square 96, A=2, gmres", mesh="square", n=96, S="nonsymmetric"),
        # the total-pressure solver with its default theta
        _case("cube 24, A=2, total pressure", n=24, theta=0.5, form="total", rtol=1e-12),
        # independent instances of different sizes and parameters advanced together
        _case("batch 24 x cube 6..16", call="batch", n=16, n_lo=6, count=24),
        # gradient of a pressure misfit with respect to the permeability of every cell
        _case("adjoint 16, A=2, 3 steps", call="adjoint", n=16, K="cells", steps=3, rtol=1e-12),
        # a posteriori error indicators of a step
        _case("estimate 24, A=2", call="estimate", n=24, precision="fp64"),
        # assembly, right-hand side and residual alone, as a program with its own solver uses them
        _case("operator 33, A=4", call="operator", n=33, J=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["loop", "loop", "loop", "loop", "step", "batch", "adjoint", "estimate", "operator"])
    J = rng.choice([1, 2, 3, 4])
    theta = rng.choice([1.0, 1.0, 0.5])
    if call == "batch":
        lo = rng.randint(3, 7)
        return _case(None, call=call, n=lo + rng.randint(0, 8), n_lo=lo, count=rng.randint(3, 30), theta=theta)
    if call == "adjoint":
        return _case(None, call=call, n=_log_int(rng, 4, 18), K="cells", steps=rng.choice([2, 3]), theta=theta,
                     rtol=1e-12)
    if call == "estimate":
        return _case(None, call=call, n=_log_int(rng, 3, 28), J=J, precision="fp64", theta=theta)
    if call == "operator":
        return _case(None, call=call, n=_log_int(rng, 3, 36), J=J, theta=theta,
                     K=rng.choice(["constant", "cells"]))
    if call == "step":
        return _case(None, call=call, n=_log_int(rng, 3, 26), J=J, theta=theta,
                     boundary=rng.choice(["dirichlet", "mixed"]))
    what = rng.choice(["cube", "cube", "cube", "fp64", "shell", "square", "total"])
    if what == "fp64":
        return _case(None, n=_log_int(rng, 3, 26), J=J, precision="fp64", theta=theta)
    if what == "shell":
        return _case(None, mesh="shell", n=_log_int(rng, 3, 11), J=J, K=rng.choice(["constant", "cells"]),
                     theta=theta)
    if what == "square":
        return _case(None, mesh="square", n=_log_int(rng, 8, 130), J=2, theta=theta,
                     S=rng.choice(["symmetric", "nonsymmetric"]), precision=rng.choice(["mixed", "fp64"]))
    if what == "total":
        return _case(None, n=_log_int(rng, 3, 26), J=rng.choice([1, 2, 3]), theta=0.5, form="total", rtol=1e-12)
    return _case(None, n=_log_int(rng, 3, 48), J=J, theta=theta)


# --- problems ------------------------------------------------------------------------

_meshes = {}


def _mesh(kind, n):
    """Meshes are made once per size: a program reads its mesh once, too."""
    key = (kind, n)
    if key not in _meshes:
        m = MESHES[kind](n)
        m.boundary_facets()
        _meshes[key] = m
    return _meshes[key]


def _materials(case, rng):
    """The material sets of the framework's cube workloads; J other than 2 and 4 as in its tests."""
    J = case["J"]
    if case["mesh"] == "square":
        S = ((0.0, 2.0), (1.0, 0.0)) if case["S"] == "nonsymmetric" else ((0.0, 1.5), (1.5, 0.0))
        E, nu = 3 * 0.479 * 100, 0.479
        return dict(J=2, c=(0.3, 0.4), alpha=(0.4, 0.6), K=(0.2, 0.3), S=S, E=E, nu=nu), 0.02
    E, nu = convert_to_E_nu(1.0e3, 1.0e4)
    S = np.zeros((J, J))
    if J == 2:
        alpha, c, K, dt = (0.5, 0.5), (1e-4, 1e-4), (1e-3, 1e-2), 0.0125
        S[:] = [[0.0, 0.1], [0.1, 0.0]]
    elif J == 4:
        alpha, c, K, dt = (0.25,) * 4, (1e-4,) * 4, (1e-4, 1e-3, 1e-2, 1e-1), 0.01
        S[:] = 1e-2
        np.fill_diagonal(S, 0.0)
    else:
        alpha = tuple(0.3 + 0.1 * a for a in range(J))
        c, K, dt = tuple(1e-3 * (a + 1) for a in range(J)), tuple(10.0 ** (-3 + a) for a in range(J)), 0.02
    if case["form"] == "total":
        E, nu = 3.0e3, 0.48
    if case["K"] == "cells":
        nc = _mesh(case["mesh"], case["n"]).num_cells()
        K = tuple(10.0 ** rng.normal(math.log10(k), 0.5, size=nc) for k in K)
    return dict(J=J, E=E, nu=nu, alpha=alpha, c=c, K=K, S=tuple(map(tuple, S))), dt


def _pulse(amp, phase):
    """Boundary pressure: a pulse over the cycle, sloped along x."""
    return lambda x, t: amp * (math.sin(2 * math.pi * (t + phase)) * x[:, 0] + 0.1 * x[:, 1])


def _problem(case, rng):
    mesh = _mesh(case["mesh"], case["n"])
    params, dt = _materials(case, rng)
    p = MPETProblem(mesh, Constant(0.0), params=params)
    J = params["J"]
    on_boundary = CompiledSubDomain.on_boundary()
    on_boundary.mark(p.momentum_boundary_markers, DIRICHLET)
    for a in range(J):
        on_boundary.mark(p.continuity_boundary_markers[a], DIRICHLET)
    amp = rng.uniform(0.5, 1.5, size=J) * np.arange(1, J + 1)
    phase = rng.uniform(0.0, 0.2, size=J)
    p.p_bar = [Expression(_pulse(float(amp[a]), float(phase[a]))) for a in range(J)]
    if case["boundary"] == "mixed":
        right = CompiledSubDomain(lambda x: np.abs(x[:, 0] - 1.0) < 1e-12)
        top = CompiledSubDomain(lambda x: np.abs(x[:, 1] - 1.0) < 1e-12)
        right.mark(p.momentum_boundary_markers, NEUMANN)
        right.mark(p.continuity_boundary_markers[0], NEUMANN)
        top.mark(p.continuity_boundary_markers[0], ROBIN)
        s0, i0, b0 = (float(v) for v in rng.uniform(0.5, 1.5, size=3))
        p.s = Expression(lambda x, t, n: s0 * (1.0 + t) * n * x[:, :1])
        p.I[0] = Expression(lambda x, t: i0 * (x[:, 1] + t))
        p.beta[0] = Expression(lambda x, t: b0 + x[:, 2])
        p.p_robin[0] = Expression(lambda x, t: x[:, 0] + t)
        p.f = Expression(lambda x, t: (1.0 + t) * x * (1.0 - x))
        p.g[J - 1] = Expression(lambda x, t: math.cos(t) * x[:, 0] * x[:, 2])
    return p, dt


def _params(case, dt):
    return dict(dt=dt, T=1e9, theta=case["theta"], precision=case["precision"], rtol=case["rtol"])


def _batch_sizes(case):
    r = np.random.default_rng(case["count"])
    return [int(v) for v in r.integers(case["n_lo"], case["n"] + 1, size=case["count"])]


def _batch_problems(case, rng):
    """Instances with log-uniform K, c and S12, as in the batched workload."""
    lu = lambda lo, hi: float(10.0 ** rng.uniform(math.log10(lo), math.log10(hi)))  # noqa: E731
    out = []
    for n in _batch_sizes(case):
        p, _ = _problem(dict(case, n=n), rng)
        s12 = lu(1e-3, 1.0)
        p.params.update(K=(lu(1e-5, 1e-1), lu(1e-5, 1e-1)), c=(lu(1e-5, 1e-3), lu(1e-5, 1e-3)),
                        S=((0.0, s12), (s12, 0.0)))
        out.append(p)
    return out, 0.02


def _smooth(solver, gen, scale=1e-2):
    """A smooth state with some noise, from the generator."""
    x = torch.randn(solver.N, generator=gen, dtype=torch.float64, device=solver.device)
    t = torch.linspace(0.0, 20.0, solver.N, dtype=torch.float64, device=solver.device)
    return scale * (torch.sin(t) + 0.1 * x)


def prepare(case, seed):
    gc.collect()  # solvers that the program has dropped give their memory back first
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    call = case["call"]
    if call == "estimate":
        problem, dt = _problem(case, rng)
        params = AdaptiveMPETSolver.default_params()
        params["MPETSolver"].update(_params(case, dt))
        solver = AdaptiveMPETSolver(problem, Constant((0.0,) * 3), params)
        solver.inner_solver.up_.assign(_smooth(solver.inner_solver, gen))
        solver.inner_solver.up.assign(_smooth(solver.inner_solver, gen))
        return dict(call=call, solver=solver)
    if call == "batch":
        problems, dt = _batch_problems(case, rng)
        solver = MPETBatchSolver(problems, _params(case, dt))
    else:
        problem, dt = _problem(case, rng)
        cls = MPETTotalPressureSolver if case["form"] == "total" else MPETSolver
        solver = cls(problem, _params(case, dt))
    state = dict(call=call, solver=solver, dt=dt, t0=0.0)
    if call in ("loop", "batch", "step"):
        # the loop has taken its first step: matrix, preconditioner and a state exist
        for _ in solver.solve_direct():
            break
        solver.up_.assign(solver.up)
        state["t0"] = dt
    elif call == "adjoint":
        x = torch.as_tensor(solver.problem.mesh.coordinates(), device=solver.device)
        amp = torch.as_tensor(rng.uniform(0.02, 0.1, size=solver.J), device=solver.device)
        state.update(K=solver._K_cells.clone(), steps=case["steps"], up0=torch.zeros_like(solver.up.vector()),
                     target=amp[:, None] * torch.sin(math.pi * x[:, 0]) * x[:, 1])
    else:
        state.update(up=_smooth(solver, gen), x=_smooth(solver, gen), b=torch.empty_like(solver.up.vector()),
                     r=torch.empty_like(solver.up.vector()), y=torch.empty_like(solver.up.vector()),
                     norms=np.zeros(2))
        solver.problem.time.assign(dt)
        solver._set_bc_values(dt)
        solver._set_sources(dt, dt)
    return state


def run(state):
    call, solver = state["call"], state["solver"]
    if call == "estimate":
        return list(solver.indicators())
    dt = state["dt"]
    if call in ("loop", "batch"):
        solver.problem.time.assign(state["t0"])
        solver.advance(dt)
        return solver.up.vector()
    if call == "step":
        solver.problem.time.assign(state["t0"])
        solver.step(dt)
        return solver.up.vector()
    if call == "adjoint":
        K = state["K"].clone().requires_grad_()
        loss = pressure_misfit(solver, K, state["target"], state["steps"], t0=0.0, up0=state["up0"])
        loss.backward()
        return [loss.detach(), K.grad]
    ctx, ptr = solver.ctx, _lib._ptr
    ctx.call("mpet_assemble", dt, 1)
    ctx.call("mpet_rhs", dt, ptr(state["up"]), ptr(state["b"]))
    ctx.call("mpet_residual", ptr(state["b"]), ptr(state["x"]), ptr(state["r"]), ptr(state["norms"]))
    ctx.call("mpet_spmv", 0, ptr(state["x"]), ptr(state["y"]))
    return [state["b"], state["r"], state["y"], state["norms"]]


# --- what a pass cannot do without -----------------------------------------------------


def _counts(case):
    """(vertices, P2 nodes, cells, dim) of a case's mesh or meshes."""
    def cube(n):
        return (n + 1) ** 3, (2 * n + 1) ** 3, 6 * n ** 3
    if case["call"] == "batch":
        return tuple(sum(v) for v in zip(*map(cube, _batch_sizes(case)))) + (3,)
    n = case["n"]
    if case["mesh"] == "square":
        return (n + 1) ** 2, (2 * n + 1) ** 2, 2 * n * n, 2
    if case["mesh"] == "shell":
        shell = lambda na, nr: (6 * na * na + 2) * (nr + 1)  # noqa: E731
        return shell(2 * n, n), shell(4 * n, 2 * n), 144 * n ** 3, 3
    return cube(n) + (3,)


def work(case):
    """The mesh, the per-cell data and the state read once, the result written once; as flops
    one application of the element operators (the least that any solve or product does)."""
    nv, nn, nc, d = _counts(case)
    J = case["J"] + (1 if case["form"] == "total" else 0)
    N = d * nn + J * nv
    mesh = 8 * d * nv + 4 * (d + 1) * nc + (8 * J * nc if case["K"] == "cells" else 0)
    ne = d * (10 if d == 3 else 6) + J * (d + 1)
    flops = 2.0 * ne * ne * nc
    call = case["call"]
    if call == "adjoint":
        s = case["steps"]
        return {"bytes": mesh + 2 * s * 16 * N + 8 * J * nc, "flops": 2 * s * flops}
    if call == "estimate":
        return {"bytes": mesh + 16 * N + 24 * nc, "flops": flops}
    if call == "operator":
        return {"bytes": mesh + 40 * N, "flops": 4 * flops}
    return {"bytes": mesh + 16 * N, "flops": flops * (2 if call == "step" else 1)}


# --- the same outputs from FP64 algebra --------------------------------------------------


class _Elements:
    """P2 x P1 element matrices of the MPET form on tetrahedra, by a four-point rule that is
    exact for them, in the framework's DOF order (vertices, then edges by their end points;
    u node-interleaved, then the networks)."""

    EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]

    def __init__(self, problem, dt, theta, device):
        f64 = dict(dtype=torch.float64, device=device)
        mesh, prm = problem.mesh, problem.params
        X = torch.as_tensor(mesh.coordinates(), **f64)
        C = torch.as_tensor(np.asarray(mesh.cells(), dtype=np.int64), device=device)
        nv, nc = X.shape[0], C.shape[0]
        J = int(prm["J"])
        key = torch.stack([torch.minimum(C[:, a], C[:, b]) * nv + torch.maximum(C[:, a], C[:, b])
                           for a, b in self.EDGES], 1)
        uniq, inv = torch.unique(key, return_inverse=True)
        nn = nv + uniq.numel()
        nodes = torch.cat([C, nv + inv], 1)
        Jm = torch.stack([X[C[:, k]] - X[C[:, 0]] for k in (1, 2, 3)], 2)
        vol = torch.linalg.det(Jm).abs() / 6.0
        G = torch.linalg.inv(Jm)                                  # rows: grad lambda_1..3
        G = torch.cat([-G.sum(1, keepdim=True), G], 1)            # nc x 4 x 3
        mu, lmbda = (float(v) for v in problem.lame())
        K = [torch.as_tensor(np.broadcast_to(np.asarray(k, dtype=np.float64), (nc,)).copy(), **f64) for k in prm["K"]]
        S = torch.tensor([[float(v) for v in row] for row in prm["S"]], **f64)
        alpha = [float(v) for v in prm["alpha"]]
        c = [float(v) for v in prm["c"]]
        nu, ne = 30, 30 + 4 * J
        A = torch.zeros(nc, ne, ne, **f64)
        B = torch.zeros(nc, 4 * J, ne, **f64)
        qa, qb = 0.5854101966249685, 0.1381966011250105
        for q in range(4):
            lam = torch.full((4,), qb, **f64)
            lam[q] = qa
            w = vol / 4.0
            gp = torch.cat([torch.stack([(4 * lam[v] - 1) * G[:, v] for v in range(4)], 1),
                            torch.stack([4 * (lam[a] * G[:, b] + lam[b] * G[:, a]) for a, b in self.EDGES], 1)], 1)
            dot = torch.einsum("cik,cjk->cij", gp, gp)
            uu = mu * torch.einsum("cij,kl->cikjl", dot, torch.eye(3, **f64))
            uu = uu + mu * torch.einsum("cil,cjk->cikjl", gp, gp) + lmbda * torch.einsum("cik,cjl->cikjl", gp, gp)
            A[:, :nu, :nu] += w[:, None, None] * uu.reshape(nc, nu, nu)
            div = gp.reshape(nc, nu)
            for a in range(J):
                s = slice(nu + 4 * a, nu + 4 * a + 4)
                up = -alpha[a] * w[:, None, None] * div[:, :, None] * lam[None, None, :]
                A[:, :nu, s] += up
                A[:, s, :nu] += up.transpose(1, 2)
                B[:, 4 * a: 4 * a + 4, :nu] += up.transpose(1, 2)
        M = vol[:, None, None] / 20.0 * (torch.ones(4, 4, **f64) + torch.eye(4, **f64))
        L = vol[:, None, None] * torch.einsum("cik,cjk->cij", G, G)
        for a in range(J):
            sa = slice(nu + 4 * a, nu + 4 * a + 4)
            ra = slice(4 * a, 4 * a + 4)
            A[:, sa, sa] -= c[a] * M + dt * theta * K[a][:, None, None] * L
            B[:, ra, sa] += -c[a] * M + dt * (1 - theta) * K[a][:, None, None] * L
            for b in range(J):
                sb = slice(nu + 4 * b, nu + 4 * b + 4)
                A[:, sa, sa] -= dt * theta * S[a, b] * M
                A[:, sa, sb] += dt * theta * S[a, b] * M
                B[:, ra, sa] += dt * (1 - theta) * S[a, b] * M
                B[:, ra, sb] -= dt * (1 - theta) * S[a, b] * M
        self.A, self.B, self.J, self.nv, self.nn, self.N = A, B, J, nv, nn, 3 * nn + J * nv
        u = (3 * nodes[:, :, None] + torch.arange(3, device=device)).reshape(nc, nu)
        p = torch.cat([3 * nn + a * nv + C for a in range(J)], 1)
        self.dofs = torch.cat([u, p], 1)
        self.pdofs = p
        # Dirichlet degrees of freedom: every node of a boundary facet
        bf = torch.as_tensor(np.asarray(mesh.boundary_facets(), dtype=np.int64), device=device)
        bk = torch.cat([torch.minimum(bf[:, a], bf[:, b]) * nv + torch.maximum(bf[:, a], bf[:, b])
                        for a, b in ((0, 1), (0, 2), (1, 2))])
        bn = torch.unique(torch.cat([bf.reshape(-1), nv + torch.searchsorted(uniq, bk)]))
        bv = torch.unique(bf.reshape(-1))
        self.bc_u = (3 * bn[:, None] + torch.arange(3, device=device)).reshape(-1)
        self.bc_p = [3 * nn + a * nv + bv for a in range(J)]
        self.xv = X[bv]
        self.bc = torch.cat([self.bc_u] + self.bc_p)

    def bc_vector(self, problem, t, b):
        b[self.bc_u] = 0.0
        for a in range(self.J):
            b[self.bc_p[a]] = problem.p_bar[a].fn(self.xv, t)
        return b

    def apply(self, x):
        y = torch.zeros_like(x)
        y.index_add_(0, self.dofs.reshape(-1), torch.einsum("cij,cj->ci", self.A, x[self.dofs]).reshape(-1))
        y[self.bc] = x[self.bc]
        return y

    def rhs(self, problem, up, t1):
        b = torch.zeros_like(up)
        b.index_add_(0, self.pdofs.reshape(-1), torch.einsum("cij,cj->ci", self.B, up[self.dofs]).reshape(-1))
        return self.bc_vector(problem, t1, b)

    def diagonal(self):
        d = torch.zeros(self.N, dtype=torch.float64, device=self.A.device)
        d.index_add_(0, self.dofs.reshape(-1), torch.diagonal(self.A, dim1=1, dim2=2).reshape(-1))
        d[self.bc] = 1.0
        return d

    def dense(self):
        D = torch.zeros(self.N * self.N, dtype=torch.float64, device=self.A.device)
        idx = self.dofs[:, :, None] * self.N + self.dofs[:, None, :]
        D.index_add_(0, idx.reshape(-1), self.A.reshape(-1))
        D = D.view(self.N, self.N)
        D[self.bc] = 0.0
        D[self.bc, self.bc] = 1.0
        return D


def exact(case, seed):
    plain = case["form"] == "mpet" and case["boundary"] == "dirichlet" and case["mesh"] != "square"
    if not plain or case["call"] not in ("loop", "step", "operator"):
        return None
    if case["call"] != "operator" and (case["mesh"] != "cube" or case["n"] > 8):
        return None
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    problem, dt = _problem(case, rng)
    E = _Elements(problem, dt, case["theta"], "cuda")
    if case["call"] == "operator":
        shape = type("Shape", (), dict(N=E.N, device="cuda"))
        up, x = _smooth(shape, gen), _smooth(shape, gen)
        b = E.rhs(problem, up, dt)
        y = E.apply(x)
        d = E.diagonal().abs()
        r = b - y
        return [b, r, y, np.array([float((r / d).norm()), float((b / d).norm())])]
    D = E.dense()
    lu = torch.linalg.lu_factor(D)

    def solve(b):
        x = torch.linalg.lu_solve(*lu, b[:, None])[:, 0]
        for _ in range(2):
            x = x + torch.linalg.lu_solve(*lu, (b - D @ x)[:, None])[:, 0]
        return x

    up = solve(E.rhs(problem, torch.zeros(E.N, dtype=torch.float64, device="cuda"), dt))
    return solve(E.rhs(problem, up, 2 * dt))
