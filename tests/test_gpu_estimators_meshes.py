"""The error indicators on distorted meshes with shuffled vertex numbers (every pairing of local
vertices across a facet), from one cell column to several blocks with a partial last one, against
the estimator oracle within the bar of the structured meshes (rtol 1e-11, 1e-13 of the largest):
both evaluate the same sums in FP64, a few hundred operations each.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dim,n", [(2, 1), (2, 9), (3, 1), (3, 4)])
def test_indicators_on_shuffled_meshes(dim, n, monkeypatch):
    import waterscapes_gb300 as w
    from test_gpu_estimators import _adaptive, _oracle_indicators
    rng = np.random.default_rng(17 * dim + n)

    def shuffled(make):
        m = make(n)
        x, cells = np.asarray(m.coordinates()), np.asarray(m.cells())
        p = rng.permutation(len(x))
        y = np.empty_like(x)
        y[p] = x + rng.uniform(-0.15 / n, 0.15 / n, x.shape)
        return w.Mesh(y, p[cells])

    for name in ("UnitSquareMesh", "UnitCubeMesh"):
        make = getattr(w, name)
        monkeypatch.setattr(w, name, lambda n, make=make: shuffled(make))
    dt = 0.05
    ad, problem, data, time_ = _adaptive(dim, n, dt, 10 * dt)
    s = ad.inner_solver
    up, up_prev = (rng.standard_normal(s.N) * 1e-2 for _ in range(2))
    s.up.assign(torch.tensor(up))
    s.up_.assign(torch.tensor(up_prev))
    problem.time.assign(0.1 + dt)
    time_.assign(0.1)
    eta_p, eta_u, eta_udt, r4 = ad.indicators()
    ref = _oracle_indicators(problem, data, up, up_prev, dt, 0.1 + dt, 0.1)
    for got, want in zip((eta_p, eta_u, eta_udt), ref[:3]):
        assert np.allclose(got.cpu().numpy(), want, rtol=1e-11, atol=1e-13 * np.abs(want).max())
    assert abs(r4 - ref[3]) <= 1e-11 * abs(ref[3])
