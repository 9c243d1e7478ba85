"""The copies of the assembled values that the products read (FP32, SELL-32, node blocks), filled
when a product first needs them and with every later assembly.

A copy holds the values of the last mpet_assemble (mpetsolver.py:335-344) for every product, on
whatever stream it is issued and also where it is replayed from a CUDA graph.  Products against the
assembled FP64 values: FP64 within 1e-13 of |A||x| (rows of at most 300 entries, 300 roundings of
1.1e-16, rounded up), FP32 within 2e-5 (300 roundings of 6e-8), both in the maximum norm.
"""
import numpy as np
import pytest

from helpers import make_problem

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

VARIANTS = [(None, "fp64"), (8, "fp64"), (4, "fp64"), (0, "fp64"), (None, "mixed"), (9, "mixed"), (4, "mixed"),
            (0, "mixed")]


def _solver(precision, variant, n=5):
    from waterscapes_gb300 import MPETSolver
    problem, dt = make_problem(n, 2)
    s = MPETSolver(problem, dict(dt=dt, T=1.0, precision=precision))
    if variant is not None:
        s.ctx.call("mpet_set_spmv_variant", variant)
    return s, dt


def _matrix(s):
    import scipy.sparse as sp
    rp, ci = s.pattern()
    return sp.csr_matrix((s.matrix_values(), ci, rp), shape=(s.N, s.N))


def _vectors(s, p):
    x = torch.tensor(np.random.default_rng(4).standard_normal(s.N), device=s.device,
                     dtype=torch.float32 if p else torch.float64)
    return x, torch.full_like(x, float("nan"))


def _check(s, p, x, y):
    A = _matrix(s)
    xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
    assert (np.abs(yd - A @ xd) <= (2e-5 if p else 1e-13) * (abs(A) @ np.abs(xd)) + 1e-300).all()


@pytest.mark.parametrize("variant,precision", VARIANTS)
def test_a_captured_product_runs_on_the_last_assembly(variant, precision):
    from waterscapes_gb300 import _lib
    s, dt = _solver(precision, variant)
    side = torch.cuda.Stream()
    s.ctx.call("mpet_set_stream", side.cuda_stream)
    p = 1 if precision == "mixed" else 0
    x, y = _vectors(s, p)
    s.ctx.call("mpet_assemble", dt, 1)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):  # the first product since the set-up: its copy is filled here
        s.ctx.call("mpet_spmv", p, _lib._ptr(x), _lib._ptr(y))
    # a product and a solve that read the copy before the graph has run
    y2 = torch.full_like(y, float("nan"))
    s.ctx.call("mpet_spmv", p, _lib._ptr(x), _lib._ptr(y2))
    torch.cuda.synchronize()
    _check(s, p, x, y2)
    for f in (1.0, 3.0, 0.25):
        s.ctx.call("mpet_assemble", f * dt, 1)
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        _check(s, p, x, y)


def test_a_captured_right_hand_side_leaves_the_copy_filled():
    from waterscapes_gb300 import _lib
    s, dt = _solver("mixed", None)
    side = torch.cuda.Stream()
    s.ctx.call("mpet_set_stream", side.cuda_stream)
    up = torch.tensor(np.random.default_rng(5).standard_normal(s.N), device=s.device)
    b, b1 = torch.empty_like(up), torch.empty_like(up)
    s.ctx.call("mpet_assemble", dt, 0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        s.ctx.call("mpet_rhs", dt, _lib._ptr(up), _lib._ptr(b))
    s.ctx.call("mpet_rhs", dt, _lib._ptr(up), _lib._ptr(b1))
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(b, b1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_product_on_another_stream_finds_the_copy_filled(precision):
    from waterscapes_gb300 import _lib
    s, dt = _solver(precision, None, n=8)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    p = 1 if precision == "mixed" else 0
    x, y = _vectors(s, p)
    y2 = torch.full_like(y, float("nan"))
    torch.cuda.synchronize()
    s.ctx.call("mpet_set_stream", a.cuda_stream)
    for f in (1.0, 2.0):
        s.ctx.call("mpet_assemble", f * dt, 1)
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)  # what is issued on a now starts some 10 ms later
        s.ctx.call("mpet_spmv", p, _lib._ptr(x), _lib._ptr(y))
        s.ctx.call("mpet_set_stream", b.cuda_stream)
        s.ctx.call("mpet_spmv", p, _lib._ptr(x), _lib._ptr(y2))
        b.synchronize()
        _check(s, p, x, y2)
        a.synchronize()
        _check(s, p, x, y)
        s.ctx.call("mpet_set_stream", a.cuda_stream)


def test_columns_zeroed_by_apply_symmetric_reach_the_copies():
    from waterscapes_gb300 import _lib
    s, dt = _solver("mixed", None)
    s.ctx.call("mpet_assemble", dt, 1)
    for p in (0, 1):
        x, y = _vectors(s, p)
        s.ctx.call("mpet_spmv", p, _lib._ptr(x), _lib._ptr(y))
    b, xbc = torch.zeros(s.N, device=s.device, dtype=torch.float64), torch.ones(s.N, device=s.device,
                                                                               dtype=torch.float64)
    s.ctx.call("mpet_apply_symmetric", _lib._ptr(b), _lib._ptr(xbc))
    for p in (0, 1):
        x, y = _vectors(s, p)
        s.ctx.call("mpet_spmv", p, _lib._ptr(x), _lib._ptr(y))
        torch.cuda.synchronize()
        _check(s, p, x, y)
