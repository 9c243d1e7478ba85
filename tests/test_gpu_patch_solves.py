"""Solves whose inner products are formed element by element, on the paths that differ in what
surrounds them: non-symmetric transfer (GMRES), batches whose instances converge at different
iterations, zeroed Dirichlet columns, a batch declared after the assembly.

The mixed-precision solves refine to 1e-11 in FP64 residuals, so a state agrees with the direct
solution, or with the same solve by the stored matrix, within 1e-8 (mpetsolver.py:317-379).
"""
import ctypes

import numpy as np
import pytest

from helpers import cfg_params, make_oracle, make_problem, oracle_data

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _product_error(s):
    """Krylov product by elements against the assembled values, the worst of the row blocks."""
    import scipy.sparse as sp
    from waterscapes_gb300 import _lib
    rp, ci = s.pattern()
    A = sp.csr_matrix((s.matrix_values(), ci, rp), shape=(s.N, s.N))
    x = torch.tensor(np.random.default_rng(3).standard_normal(s.N), dtype=torch.float32, device=s.device)
    y = torch.full_like(x, float("nan"))
    used = ctypes.c_int32()
    s.ctx.call("mpet_krylov_product", _lib._ptr(x), _lib._ptr(y), ctypes.byref(used))
    torch.cuda.synchronize()
    assert used.value == 1
    xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
    err, scale = np.abs(yd - A @ xd), abs(A) @ np.abs(xd)
    return max(np.linalg.norm(err[b]) / np.linalg.norm(scale[b])
               for b in [slice(0, s.Nu)] + [slice(s.Nu + a * s.nv, s.Nu + (a + 1) * s.nv) for a in range(s.J)])


def _nonsymmetric(n, J):
    problem, dt = make_problem(n, J)
    S = np.random.default_rng(J).uniform(0.0, 50.0, (J, J))
    np.fill_diagonal(S, 0.0)
    problem.params.update(S=tuple(tuple(r) for r in S), c=tuple(0.1 * (a + 1) for a in range(J)))
    return problem, dt


@pytest.mark.parametrize("J", [2, 3])
@pytest.mark.parametrize("cells", [False, True])
def test_non_symmetric_transfer_in_the_product(J, cells):
    from waterscapes_gb300 import MPETSolver, _lib
    problem, dt = _nonsymmetric(4, J)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed"))
    s.ctx.call("mpet_set_element_product", 1)
    if cells:
        nc = problem.mesh.num_cells()
        S = torch.tensor(np.random.default_rng(9).uniform(0.0, 50.0, (J, J, nc)), device=s.device)
        s.ctx.call("mpet_set_cell_coefficients", None, _lib._ptr(S))
    s.ctx.call("mpet_assemble", dt, 0)
    assert _product_error(s) <= 2e-6


def test_gmres_steps_with_the_element_product():
    from waterscapes_gb300 import MPETSolver
    problem, dt = _nonsymmetric(4, 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed", rtol=1e-11))
    s.ctx.call("mpet_set_element_product", 1)
    om = make_oracle(problem)
    ref, t = np.zeros(om.dm.N), 0.0
    for h in (dt, 3.0 * dt, dt):  # the captured product takes each assembly's coefficients
        assert s.step(h).status == 0
        s.up_.assign(s.up)
        ref = om.step(ref, t, h, oracle_data(2))
        t += h
        assert _rel(s.up.vector().cpu().numpy(), ref) <= 1e-8
        assert _product_error(s) <= 2e-6


@pytest.mark.parametrize("sizes", [(2, 4, 3, 6), (2, 9, 3)])
def test_instances_that_converge_apart(sizes):
    """Permeabilities from 1e-4 to 10: converged instances' patches give zero rows while the others go on;
    each instance's state is that of its own direct solve."""
    from waterscapes_gb300 import MPETBatchSolver
    problems = []
    for i, n in enumerate(sizes):
        p, _ = make_problem(n, 2)
        p.params.update(K=(10.0 ** (-4 + 5 * i / (len(sizes) - 1)), 1e-2), c=(1e-4, 1e-3))
        problems.append(p)
    dt, out = 0.02, []
    for mode in (1, 0):
        s = MPETBatchSolver(problems, dict(dt=dt, T=1.0, precision="mixed", rtol=1e-11))
        s.ctx.call("mpet_set_element_product", mode)
        for p in problems:
            p.time.assign(0.0)
        for _ in range(2):
            s.step(dt)
            s.up_.assign(s.up)
        out.append(s.up.vector().cpu().numpy())
    assert np.isfinite(out[0]).all()
    assert _rel(out[0], out[1]) <= 1e-8


def test_solve_with_zeroed_dirichlet_columns():
    """mpet_apply_symmetric zeroes columns that the element product still has: the inner vectors are zero
    there, so the solve is the same."""
    from waterscapes_gb300 import MPETSolver, _lib
    out = []
    for mode in (1, 0):
        problem, dt = make_problem(5, 2)
        s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed", rtol=1e-11))
        s.ctx.call("mpet_set_element_product", mode)
        s.step(dt)
        x1 = s.up.vector().clone()
        prev = s.up_.vector()
        b, x = torch.empty_like(x1), prev.clone()
        s.ctx.call("mpet_rhs", dt, _lib._ptr(prev), _lib._ptr(b))
        xbc = torch.zeros_like(x1)
        for f in s._bcs:
            xbc[f["dofs"].long()] = x1[f["dofs"].long()]
        s.ctx.call("mpet_apply_symmetric", _lib._ptr(b), _lib._ptr(xbc))
        st = _lib.MpetStats()
        s.ctx.call("mpet_solve", _lib._ptr(b), _lib._ptr(x), ctypes.byref(st))
        assert st.status == 0
        assert torch.linalg.norm(x - x1) <= 1e-8 * torch.linalg.norm(x1)
        out.append(x.cpu().numpy())
    assert _rel(out[0], out[1]) <= 1e-8


def test_batch_declared_after_an_assembly():
    from waterscapes_gb300 import CompiledSubDomain, Constant, Mesh, MPETProblem, MPETSolver, UnitCubeMesh, _lib
    a, b = UnitCubeMesh(3), UnitCubeMesh(4)
    nva = a.num_vertices()
    mesh = Mesh(np.concatenate([a.coordinates(), b.coordinates() + [2.0, 0.0, 0.0]]),
                np.concatenate([a.cells(), b.cells() + nva]))
    params, dt = cfg_params(2)
    problem = MPETProblem(mesh, Constant(0.0), params=params)
    CompiledSubDomain.on_boundary().mark(problem.momentum_boundary_markers, 0)
    for k in range(2):
        CompiledSubDomain.on_boundary().mark(problem.continuity_boundary_markers[k], 0)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed", rtol=1e-11))
    s.ctx.call("mpet_set_element_product", 1)
    s.ctx.call("mpet_assemble", dt, 1)
    s.ctx.call("mpet_setup_preconditioner", dt)
    rhs = torch.tensor(np.random.default_rng(2).standard_normal(s.N), device=s.device)
    for f in s._bcs:
        rhs[f["dofs"].long()] = 0.0
    x1, x2 = torch.zeros_like(rhs), torch.zeros_like(rhs)
    st = _lib.MpetStats()
    s.ctx.call("mpet_solve", _lib._ptr(rhs), _lib._ptr(x1), ctypes.byref(st))
    inst = np.concatenate([np.zeros(nva), np.ones(b.num_vertices())]).astype(np.int32)
    s.ctx.call("mpet_set_batch", 2, _lib._ptr(inst))
    s.ctx.call("mpet_setup_preconditioner", dt)  # without another assembly
    assert _product_error(s) <= 2e-6
    s.ctx.call("mpet_solve", _lib._ptr(rhs), _lib._ptr(x2), ctypes.byref(st))
    assert st.status == 0
    assert torch.linalg.norm(x2 - x1) <= 1e-8 * torch.linalg.norm(x1)
