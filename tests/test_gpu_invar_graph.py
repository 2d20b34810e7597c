"""FAME_OP_INVAR runs one recorded graph: it serves every wave vector, permittivity, tolerance and product
cap, and is recorded again only when the workspace changes."""
import numpy as np
import pytest

import fame_b200 as fb
from fixtures import load_pre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _ctx(B):
    par = load_pre("fcc16")
    ctx = fb.Context.from_par(par)
    ctx.set_eps(B)
    return ctx


def _apply(ctx, k, x, tol, maxit):
    nd = fb.reduced_size(ctx._lat, k)
    xd = torch.from_numpy(x[:2 * nd].copy()).to("cuda")
    y = torch.zeros(2 * nd, dtype=torch.complex128, device="cuda")
    ctx.apply(fb.OP_INVAR, k, xd, y, fb.FP64, fb.solver_params(ls_tol=tol, ls_maxit=maxit))
    return y.cpu().numpy()


def test_one_graph_serves_every_call():
    par = load_pre("fcc16")
    N = int(np.prod(par["grid"]))
    rng = np.random.default_rng(3)
    x = rng.standard_normal(2 * N) + 1j * rng.standard_normal(2 * N)
    eps = [rng.uniform(1.0, 13.0, 3 * N) for _ in range(2)]
    ks = [np.array([0.11, -0.23, 0.31]), np.zeros(3), np.array([0.3, 0.1, -0.2])]
    ctx = _ctx(eps[0])
    _apply(ctx, ks[0], x, 1e-12, 1000)
    before = ctx.get_option("graphs_recorded")
    calls = [(0, 0, 1e-12, 1000), (0, 1, 1e-12, 1000), (0, 2, 1e-3, 1000), (1, 0, 1e-8, 1000), (1, 1, 1e-12, 3), (0, 0, 1e-12, 1000)]
    for e, q, tol, maxit in calls:
        ctx.set_eps(eps[e])
        fresh = _ctx(eps[e])
        assert np.array_equal(_apply(ctx, ks[q], x, tol, maxit), _apply(fresh, ks[q], x, tol, maxit)), (e, q, tol, maxit)
        fresh.close()
    assert ctx.get_option("graphs_recorded") == before
    # a solve regrows the workspace: recorded once more, with the same results
    ctx.solve(ks[0].reshape(1, 3), nwant=4, nstep=20, es_tol=1e-8, ls_tol=1e-8)
    y = _apply(ctx, ks[2], x, 1e-12, 1000)
    fresh = _ctx(eps[0])
    assert np.array_equal(y, _apply(fresh, ks[2], x, 1e-12, 1000))
    fresh.close()
    ctx.close()
