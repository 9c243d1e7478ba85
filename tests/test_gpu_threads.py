"""Contexts of different sizes in threads of their own (one context per host thread): their launches
share the process's kernels, not each other's limits."""
import ctypes
import threading

import numpy as np
import pytest

from helpers import make_oracle, make_problem, oracle_data

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_contexts_of_two_sizes_solve_side_by_side():
    from waterscapes_gb300 import MPETSolver
    sizes = (3, 9)
    solvers = []
    for n in sizes:
        problem, dt = make_problem(n, 2)
        s = MPETSolver(problem, dict(dt=dt, T=1.0, precision="mixed", rtol=1e-11))
        st = torch.cuda.Stream()
        s.ctx.call("mpet_set_stream", st.cuda_stream)
        s.ctx.call("mpet_set_element_product", 1)
        s.ctx.call("mpet_set_row_tiles", 1)
        solvers.append((s, st, dt, problem))
    torch.cuda.synchronize()
    errors, results = [], {}

    def work(k):
        s, st, dt, _ = solvers[k]
        try:
            for rep in range(6):
                s.ctx.call("mpet_update_params", ctypes.byref(s._prm))  # everything is set up again
                s._assembled_dt = s._prec_dt = None
                s.up_.vector().zero_()
                s.problem.time.assign(0.0)
                with torch.cuda.stream(st):
                    s.step(dt)
                st.synchronize()
            results[k] = s.up.vector().cpu().numpy()
        except Exception as e:  # noqa: BLE001
            errors.append((k, e))

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors
    for k in range(len(sizes)):
        s, _, dt, problem = solvers[k]
        om = make_oracle(problem)
        ref = om.step(np.zeros(om.dm.N), 0.0, dt, oracle_data(2))
        assert np.linalg.norm(results[k] - ref) <= 1e-8 * np.linalg.norm(ref)
