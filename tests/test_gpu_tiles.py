"""Level operators of the preconditioner by row tiles against the CSR kernels.

The same operators with other summation orders: one preconditioner application agrees to
round-off (FP64: 1e-12; FP32: 1e-4 relative, as for the other kernels of these levels), and a
step with the tiles is the oracle's step.  The tiles are forced on every level, so the cases
cover each tile height (32 to 256 rows), ragged last tiles, levels smaller than a tile, wide
(three or two components) and scalar vectors, and both precisions.
"""
import numpy as np
import pytest

from helpers import make_oracle, make_problem, oracle_data

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _apply(s, mode, dt):
    from waterscapes_gb300 import _lib
    s.ctx.call("mpet_set_row_tiles", mode)
    s.ctx.call("mpet_setup_preconditioner", dt)
    if mode == 0:
        s.ctx.call("mpet_set_hierarchy_spmv_variant", 0)
    else:
        va = np.zeros(16, np.int32)
        s.ctx.call("mpet_get_amg_variants", 0, _lib._ptr(va), None, None)
        assert va[0] in (16, 64)
    mixed = s.params["precision"] == "mixed"
    dtype = torch.float32 if mixed else torch.float64
    r = torch.tensor(np.random.default_rng(6).standard_normal(s.N), dtype=dtype, device=s.device)
    z = torch.full_like(r, float("nan"))
    s.ctx.call("mpet_apply_preconditioner", 1 if mixed else 0, _lib._ptr(r), _lib._ptr(z))
    torch.cuda.synchronize()
    return z.double().cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("mesh,n", [("cube", 1), ("cube", 5), ("cube", 9), ("cube", 17), ("square", 40), ("shell", 3)])
def test_tiles_match_csr_levels(mesh, n, precision):
    from waterscapes_gb300 import (CompiledSubDomain, Constant, EllipsoidShellMesh, MPETProblem, MPETSolver,
                                   UnitSquareMesh)
    from helpers import cfg_params
    if mesh == "cube":
        problem, dt = make_problem(n, 2)
    else:
        params, dt = cfg_params(2)
        problem = MPETProblem(UnitSquareMesh(n) if mesh == "square" else EllipsoidShellMesh(n), Constant(0.0),
                              params=params)
        CompiledSubDomain.on_boundary().mark(problem.momentum_boundary_markers, 0)
        for a in range(2):
            CompiledSubDomain.on_boundary().mark(problem.continuity_boundary_markers[a], 0)
    s = MPETSolver(problem, dict(dt=dt, T=dt, precision=precision, rtol=1e-11, amg_coarse_size=60))
    s.ctx.call("mpet_set_prec_matrix_free", 0)
    s.ctx.call("mpet_assemble", dt, 1)
    z0 = _apply(s, 0, dt)
    z1 = _apply(s, 1, dt)
    tol = 1e-12 if precision == "fp64" else 1e-4
    assert np.linalg.norm(z1 - z0) <= tol * np.linalg.norm(z0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_step_with_tiles_matches_oracle(precision):
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(5, 2)
    s = MPETSolver(problem, dict(dt=dt, T=dt, precision=precision, rtol=1e-11))
    s.ctx.call("mpet_set_row_tiles", 1)
    assert s.step(dt).status == 0
    om = make_oracle(problem)
    x_ref = om.step(np.zeros(om.dm.N), 0.0, dt, oracle_data(2))
    x = s.up.vector().cpu().numpy()
    assert np.linalg.norm(x - x_ref) <= 1e-8 * np.linalg.norm(x_ref)


def test_batch_with_tiles_matches_batch_without():
    """Converged instances' tiles are skipped; the results of the others do not change."""
    from waterscapes_gb300 import MPETBatchSolver
    out = []
    for mode in (0, 1):
        problems = []
        for i, n in enumerate((2, 4, 3, 6)):
            p, _ = make_problem(n, 2)
            p.params.update(K=(10.0 ** (-4 + i), 1e-2), c=(1e-4, 1e-3))
            problems.append(p)
        s = MPETBatchSolver(problems, dict(dt=0.02, T=1.0, precision="mixed", rtol=1e-11))
        s.ctx.call("mpet_set_row_tiles", mode)
        s.step(0.02)
        out.append(s.up.vector().clone())
    assert torch.linalg.norm(out[1] - out[0]) <= 1e-8 * torch.linalg.norm(out[0])
