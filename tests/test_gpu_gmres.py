"""The GMRES iteration (captured product and preconditioner, device-side orthogonalisation) against
the oracle's direct solution, where its pieces meet: one block and many blocks of the reductions,
restarts after 3 and 30 vectors and none (64), both precisions, a second solve that reuses the
captured graph.

Tolerance 1e-8: the solver stops at a preconditioned residual of 1e-11 of its start, and the step
tests of these small problems hold it against the direct solution to 1e-8.
"""
import numpy as np
import pytest

import mms
from helpers import make_oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,restart,precision", [(6, 3, "fp64"), (6, 3, "mixed"), (24, 30, "fp64"), (24, 30, "mixed"),
                                                 (24, 64, "mixed")])
def test_gmres_restarts_match_direct_solution(n, restart, precision):
    from test_gpu_2d import REF_PARAMS, _problem_2d
    from waterscapes_gb300 import MPETSolver
    data, _ = mms.exact_solutions(REF_PARAMS, 2)
    problem = _problem_2d(n, REF_PARAMS, data)
    dt, t0 = 0.05, 0.1
    s = MPETSolver(problem, dict(dt=dt, T=10 * dt, theta=1.0, precision=precision, rtol=1e-11, gmres_restart=restart))
    om = make_oracle(problem, 1.0)
    rng = np.random.default_rng(5)
    for _ in range(2):
        up_prev = rng.standard_normal(om.dm.N) * 1e-2
        x_ref = om.step(up_prev, t0, dt, data)
        s.up_.assign(torch.tensor(up_prev))
        problem.time.assign(t0)
        assert s.step(dt).status == 0
        x = s.up.vector().cpu().numpy()
        assert np.linalg.norm(x - x_ref) <= 1e-8 * np.linalg.norm(x_ref)
