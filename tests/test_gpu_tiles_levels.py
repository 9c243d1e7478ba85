"""Row tiles where a hierarchy has one level only: the displacement level is the coarsest one, solved
by its dense inverse, and its vectors stay in the order of the rows."""
import numpy as np
import pytest

from helpers import make_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("setup", ["device", "host"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_single_level_keeps_its_order(precision, setup):
    """343 P2 nodes, at most 500 on the coarsest level, no P1 embedding above it: one application of the
    preconditioner with tiles forced and without agrees to round-off (the same dense product)."""
    from waterscapes_gb300 import MPETSolver, _lib
    problem, dt = make_problem(3, 2)
    s = MPETSolver(problem, dict(dt=dt, T=dt, precision=precision, amg_p2_to_p1=False, amg_setup=setup))
    s.ctx.call("mpet_set_prec_matrix_free", 0)
    s.ctx.call("mpet_assemble", dt, 1)
    mixed = precision == "mixed"
    r = torch.tensor(np.random.default_rng(6).standard_normal(s.N), device=s.device,
                     dtype=torch.float32 if mixed else torch.float64)
    z = []
    for mode in (0, 1):
        s.ctx.call("mpet_set_row_tiles", mode)
        s.ctx.call("mpet_setup_preconditioner", dt)
        assert len(s.amg_info(0)[0]) == 1
        z.append(torch.full_like(r, float("nan")))
        s.ctx.call("mpet_apply_preconditioner", int(mixed), _lib._ptr(r), _lib._ptr(z[-1]))
        torch.cuda.synchronize()
    assert torch.linalg.norm(z[1] - z[0]) <= (1e-5 if mixed else 1e-13) * torch.linalg.norm(z[0])
