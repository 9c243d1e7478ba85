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
