"""The FP32 system product by patches of cells (the inner products of the mixed-precision
solves) against the assembled FP64 matrix.

Both are the operator of mpetsolver.py:196-201 with Dirichlet rows; the element product
rounds each of some 30 dependent FP32 operations per value, so the error of y = A x is at
most 2e-6 (30 roundings of 6e-8) of | A | | x | in the 2-norm, separately for the
displacement rows and each network's rows.  Sizes: one cube (fewer cells than a patch),
meshes with a ragged last patch, and each of the three patch sizes; every coefficient form
(constants, per-cell K, a batch's per-cell c, K, S), 1 to 4 and 8 networks, with and without
Dirichlet rows, and the total-pressure form.
"""
import ctypes

import numpy as np
import pytest

from helpers import make_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(s, dt, apply_bc=1, elements=1):
    import scipy.sparse as sp
    from waterscapes_gb300 import _lib
    if elements:
        s.ctx.call("mpet_set_element_product", 1)
    s.ctx.call("mpet_assemble", dt, apply_bc)
    rp, ci = s.pattern()
    A = sp.csr_matrix((s.matrix_values(), ci, rp), shape=(s.N, s.N))
    x = torch.tensor(np.random.default_rng(3).standard_normal(s.N), dtype=torch.float32, device=s.device)
    y = torch.full_like(x, float("nan"))
    used = ctypes.c_int32()
    for _ in range(2):  # (a second product finds the buffers of the first)
        s.ctx.call("mpet_krylov_product", _lib._ptr(x), _lib._ptr(y), ctypes.byref(used))
    torch.cuda.synchronize()
    assert used.value == elements
    xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
    err = np.abs(yd - A @ xd)
    scale = abs(A) @ np.abs(xd)
    blocks = [slice(0, s.Nu)] + [slice(s.Nu + a * s.nv, s.Nu + (a + 1) * s.nv) for a in range(s.J)]
    for b in blocks:
        assert np.linalg.norm(err[b]) <= 2e-6 * np.linalg.norm(scale[b])


@pytest.mark.parametrize("n,J,apply_bc", [(1, 2, 1), (2, 1, 1), (3, 3, 0), (5, 4, 1), (2, 8, 1), (11, 2, 1), (15, 1, 1),
                                          (24, 2, 1)])
def test_patch_product_constant_coefficients(n, J, apply_bc):
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(n, J)
    _check(MPETSolver(problem, dict(dt=dt, precision="mixed")), dt, apply_bc)


@pytest.mark.parametrize("J", [2, 4])
def test_patch_product_cell_permeability(J):
    from waterscapes_gb300 import CompiledSubDomain, Constant, EllipsoidShellMesh, MPETProblem, MPETSolver
    from helpers import cfg_params
    mesh = EllipsoidShellMesh(3)
    params, dt = cfg_params(J)
    rng = np.random.default_rng(5)
    params["K"] = tuple(10.0 ** rng.normal(-3.0 + a, 0.5, size=mesh.num_cells()) for a in range(J))
    problem = MPETProblem(mesh, Constant(0.0), params=params)
    CompiledSubDomain.on_boundary().mark(problem.momentum_boundary_markers, 0)
    CompiledSubDomain.on_boundary().mark(problem.continuity_boundary_markers[0], 0)  # the others: no Dirichlet rows
    _check(MPETSolver(problem, dict(dt=dt, precision="mixed")), dt)


def test_patch_product_batch_coefficients():
    from waterscapes_gb300 import MPETBatchSolver
    problems = []
    for i, n in enumerate((2, 5, 3)):
        p, dt = make_problem(n, 2)
        s12 = 0.05 * (i + 1)
        p.params.update(K=(1e-3 * (i + 1), 1e-2), c=(1e-4, 2e-4 * (i + 1)), S=((0.0, s12), (s12, 0.0)))
        problems.append(p)
    _check(MPETBatchSolver(problems, dict(dt=dt, precision="mixed")), dt)


def test_patch_product_total_pressure():
    from waterscapes_gb300 import MPETTotalPressureSolver
    problem, dt = make_problem(4, 2)
    _check(MPETTotalPressureSolver(problem, dict(dt=dt, theta=0.5, precision="mixed")), dt)


def test_coefficients_follow_the_last_assembly_and_forced_variants_stay_stored():
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(4, 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed", rtol=1e-11))
    s.ctx.call("mpet_set_element_product", 1)
    s.step(dt)          # captures the iterations with dt's coefficients
    s.step(3.0 * dt)    # another dt: assembled, preconditioned and captured again
    x = s.up.vector().clone()
    t = float(problem.time)
    ref = MPETSolver(make_problem(4, 2)[0], dict(dt=dt, T=1.0, precision="fp64", rtol=1e-12))
    ref.problem.time.assign(t - 3.0 * dt)
    ref.step(3.0 * dt)
    assert torch.linalg.norm(x - ref.up.vector()) <= 1e-8 * torch.linalg.norm(x)
    _check(s, 2.0 * dt)
    s.ctx.call("mpet_set_spmv_variant", 0)
    _check(s, dt, elements=0)


@pytest.mark.parametrize("n,J", [(3, 1), (12, 2)])
def test_robin_matrix_in_the_element_product(n, J):
    """Robin terms on one side for one network, on two sides for another; Dirichlet rows elsewhere."""
    from waterscapes_gb300 import CompiledSubDomain, Expression, MPETSolver
    problem, dt = make_problem(n, J)
    side = lambda k, v: CompiledSubDomain(lambda x: np.abs(x[:, k] - v) < 1e-12)  # noqa: E731
    side(1, 1.0).mark(problem.continuity_boundary_markers[0], 2)
    side(0, 0.0).mark(problem.continuity_boundary_markers[J - 1], 2)
    side(2, 1.0).mark(problem.continuity_boundary_markers[J - 1], 1)
    problem.beta = [Expression(lambda x, t: 150.0 + x[:, 2]) for _ in range(J)]
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed"))
    s.ctx.call("mpet_set_element_product", 1)
    s.step(dt)
    _check(s, dt)
