"""Element products (FP32, by patches of cells) under the call sequences that a program may use:
the product is that of the last mpet_assemble (mpetsolver.py:335-344) whatever came between.

Products are compared with the assembled FP64 values as in test_gpu_patch.py: at most 2e-6 of
| A | | x | in the 2-norm, for the displacement rows and each network's rows.
"""
import ctypes

import numpy as np
import pytest

from helpers import make_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check_product(s, elements, values=None):
    """Krylov product against the assembled values, by elements or not as given."""
    import scipy.sparse as sp
    from waterscapes_gb300 import _lib
    rp, ci = s.pattern()
    A = sp.csr_matrix((s.matrix_values() if values is None else values, ci, rp), shape=(s.N, s.N))
    x = torch.tensor(np.random.default_rng(3).standard_normal(s.N), dtype=torch.float32, device=s.device)
    y = torch.full_like(x, float("nan"))
    used = ctypes.c_int32()
    s.ctx.call("mpet_krylov_product", _lib._ptr(x), _lib._ptr(y), ctypes.byref(used))
    torch.cuda.synchronize()
    assert used.value == elements
    xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
    err, scale = np.abs(yd - A @ xd), abs(A) @ np.abs(xd)
    for b in [slice(0, s.Nu)] + [slice(s.Nu + a * s.nv, s.Nu + (a + 1) * s.nv) for a in range(s.J)]:
        assert np.linalg.norm(err[b]) <= 2e-6 * np.linalg.norm(scale[b])


@pytest.mark.parametrize("what", ["robin", "K"])
def test_the_coefficients_are_those_of_the_assembly(what):
    """The caller's arrays may change after mpet_assemble: the set-up of the preconditioner, which
    builds the patches, does not read them again."""
    from waterscapes_gb300 import CompiledSubDomain, MPETSolver, _lib
    problem, dt = make_problem(12, 2)  # 5.3e6 entries: elements by size
    CompiledSubDomain(lambda x: np.abs(x[:, 0]) < 1e-12).mark(problem.continuity_boundary_markers[0], 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed"))
    nf, nc = problem.mesh.num_boundary_facets(), problem.mesh.num_cells()
    a = torch.full((2, nf, 3) if what == "robin" else (2, nc), 40.0, dtype=torch.float64, device=s.device)
    if what == "robin":
        s.ctx.call("mpet_set_facet_data", 4, _lib._ptr(a))
    else:
        s.ctx.call("mpet_set_cell_permeability", _lib._ptr(a))
    s.ctx.call("mpet_assemble", dt, 1)
    a.fill_(0.5)
    torch.cuda.synchronize()
    s.ctx.call("mpet_setup_preconditioner", dt)
    _check_product(s, 1)


def test_small_cells_keep_their_terms():
    """Cells of 5e-8 (metres, say) with K dt of 1e-19 and 1e-20: entries K dt h of 5e-27 are well inside
    FP32's range, but the product of the cell's volume and K dt, 2e-42, is not."""
    from waterscapes_gb300 import Mesh, MPETProblem, MPETSolver, UnitCubeMesh, Constant, _lib
    from helpers import cfg_params
    unit = UnitCubeMesh(4)
    mesh = Mesh(unit.coordinates() * 2e-7, unit.cells())
    params, _ = cfg_params(2)
    params.update(K=(1e-17, 1e-18), c=(0.0, 0.0), S=((0.0, 0.0), (0.0, 0.0)))
    s = MPETSolver(MPETProblem(mesh, Constant(0.0), params=params), dict(dt=1e-2, precision="mixed"))
    s.ctx.call("mpet_set_element_product", 1)
    s.ctx.call("mpet_assemble", 1e-2, 1)
    import scipy.sparse as sp
    rp, ci = s.pattern()
    A = sp.csr_matrix((s.matrix_values(), ci, rp), shape=(s.N, s.N))
    x = np.random.default_rng(6).standard_normal(s.N)
    x[:s.Nu] = 0.0  # the stiffness term alone in the pressure rows
    x = torch.tensor(x, dtype=torch.float32, device=s.device)
    y = torch.full_like(x, float("nan"))
    s.ctx.call("mpet_krylov_product", _lib._ptr(x), _lib._ptr(y), None)
    torch.cuda.synchronize()
    xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
    err, scale = np.abs(yd - A @ xd), abs(A) @ np.abs(xd)
    for b in [slice(0, s.Nu)] + [slice(s.Nu + a * s.nv, s.Nu + (a + 1) * s.nv) for a in range(2)]:
        assert np.linalg.norm(err[b]) <= 2e-6 * np.linalg.norm(scale[b])


@pytest.mark.parametrize("mode", [-1, 1])
def test_a_forced_variant_stays_forced(mode):
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(12, 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed"))
    s.ctx.call("mpet_set_spmv_variant", 0)
    s.ctx.call("mpet_set_element_product", mode)
    s.ctx.call("mpet_assemble", dt, 1)
    s.ctx.call("mpet_setup_preconditioner", dt)
    _check_product(s, 0)
    s.ctx.call("mpet_assemble", 2.0 * dt, 1)
    _check_product(s, 0)


@pytest.mark.parametrize("n,elements", [(12, 1), (4, 0)])
def test_the_mode_takes_effect_at_the_next_assembly(n, elements):
    """5.3e6 and 0.2e6 entries: by size, elements and the stored copy."""
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(n, 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed"))
    s.ctx.call("mpet_set_element_product", 0)
    s.ctx.call("mpet_assemble", dt, 1)
    s.ctx.call("mpet_setup_preconditioner", dt)
    _check_product(s, 0)
    for mode, used in ((-1, elements), (1, 1), (0, 0), (-1, elements)):
        s.ctx.call("mpet_set_element_product", mode)
        s.ctx.call("mpet_assemble", dt, 1)
        _check_product(s, used)


def test_the_preconditioner_before_the_assembly():
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(12, 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed"))
    s.ctx.call("mpet_setup_preconditioner", dt)
    s.ctx.call("mpet_assemble", dt, 1)
    _check_product(s, 1)


def test_vertices_of_no_cell():
    """Their rows are empty: zero in every product (no patch holds them, so the stored copy serves), and
    one in the diagonal scaling of the residual."""
    import scipy.sparse as sp
    from waterscapes_gb300 import Constant, Mesh, MPETProblem, MPETSolver, UnitCubeMesh, _lib
    from helpers import cfg_params
    unit = UnitCubeMesh(3)
    x0, c0 = unit.coordinates(), unit.cells()
    # one before all others and two behind
    mesh = Mesh(np.concatenate([[[2.0, 0.0, 0.0]], x0, [[3.0, 0.0, 0.0], [0.0, 4.0, 1.0]]]), c0 + 1)
    params, dt = cfg_params(2)
    s = MPETSolver(MPETProblem(mesh, Constant(0.0), params=params), dict(dt=dt, precision="mixed"))
    s.ctx.call("mpet_set_element_product", 1)
    s.ctx.call("mpet_assemble", dt, 1)
    _check_product(s, 0)
    rp, ci = s.pattern()
    A = sp.csr_matrix((s.matrix_values(), ci, rp), shape=(s.N, s.N))
    d = np.abs(A.diagonal())
    x = np.random.default_rng(8).standard_normal(s.N)
    b = np.ones(s.N)
    xt, bt = (torch.tensor(v, device=s.device) for v in (x, b))
    r, norms = torch.empty_like(xt), np.zeros(2)
    s.ctx.call("mpet_residual", _lib._ptr(bt), _lib._ptr(xt), _lib._ptr(r), _lib._ptr(norms))
    dinv = 1.0 / np.where(d > 0.0, d, 1.0)
    assert (d == 0.0).sum() == 3 * (3 + 2)
    ref = [np.linalg.norm(dinv * (b - A @ x)), np.linalg.norm(dinv * b)]
    assert np.allclose(norms, ref, rtol=1e-12, atol=0.0)
