"""The batched MINRES vector kernels where their chunks and layouts change: instances of one chunk
and of several (9^3: 20,577 displacement rows, chunks of 4,096), one instance alone, the first level
in natural, spatial and tile order, the elasticity form (no packed layout).

Every instance against the same problem solved alone; tolerance 1e-8, the bar of the other batch
tests (both stop at 1e-10 of their own residual).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sizes,precision,extra,tiles", [
    ((2, 9, 3), "mixed", {}, -1), ((2, 9, 3), "fp64", {}, -1), ((5,), "mixed", {}, -1),
    ((2, 9, 3), "mixed", {"prec_u_order": "spatial"}, 0), ((2, 9, 3), "mixed", {}, 1), ((2, 9, 3), "fp64", {}, 1),
    ((2, 6, 3), "mixed", {"prec_u_form": "elasticity"}, -1)])
def test_batch_chunks(sizes, precision, extra, tiles):
    from test_gpu_batch import _instance
    from waterscapes_gb300 import MPETBatchSolver, MPETSolver
    dt = 0.02
    params = dict(dt=dt, T=2 * dt, theta=1.0, precision=precision, rtol=1e-10, **extra)

    def problems():
        return [_instance(n, (10.0 ** -(1 + i), 10.0 ** -(4 - i)), (1e-4, 1e-5), 10.0 ** (-i), 1.0 + 0.3 * i)
                for i, n in enumerate(sizes)]

    bs = MPETBatchSolver(problems(), params)
    bs.ctx.call("mpet_set_row_tiles", tiles)
    states = [[bs.instance_vector(i).cpu().numpy() for i in range(bs.ninst)] for _ in bs.solve_direct()]
    assert len(states) == 2
    for i, p in enumerate(problems()):
        for k, (up, t) in enumerate(MPETSolver(p, dict(params)).solve_direct()):
            single = up.vector().cpu().numpy()
            assert np.linalg.norm(states[k][i] - single) <= 1e-8 * np.linalg.norm(single)
