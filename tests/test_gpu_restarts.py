"""Lanczos restarts: thick restarts in mixed precision (from a solve's second restart on), slots that restart
differently often in one batch, and es_maxit as a budget of products."""
import numpy as np
import pytest

import fame_b200 as fb
from fixtures import load_pre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _ctx(name="sc16"):
    par = load_pre(name)
    ctx = fb.Context.from_par(par)
    ctx.set_material(par["binout"], par["material_num"], par["eps_in"], par["eps_out"])
    return par, ctx


# off the symmetry planes, and one at which the Krylov space converges at once beside them
KS = np.array([[0.11, -0.23, 0.31], [0.05, 0.02, -0.03], [0.37, 0.41, -0.29]])


@pytest.mark.parametrize("nwant,nstep", [(8, 12), (5, 7), (6, 20)])
def test_mixed_restarts_agree_with_fp64(nwant, nstep):
    """Frequencies within 1e-8 of FP64's (es_tol 1e-10 on the eigenvalues of A_r^-1, which are below 1),
    whatever the number of restarts, in one batch and alone."""
    _, ctx = _ctx()
    kw = dict(nwant=nwant, nstep=nstep, es_tol=1e-10, ls_tol=1e-11, es_maxit=400)
    f64 = ctx.solve(KS, precision=fb.FP64, batch=3, **kw)
    mix = ctx.solve(KS, precision=fb.MIXED, batch=3, **kw)
    one = ctx.solve(KS, precision=fb.MIXED, batch=1, **kw)
    assert f64["rc"] == fb.OK and mix["rc"] == fb.OK and one["rc"] == fb.OK
    assert np.max(np.abs(mix["freq"] - f64["freq"])) < 1e-8 * np.max(f64["freq"])
    assert np.max(np.abs(one["freq"] - f64["freq"])) < 1e-8 * np.max(f64["freq"])
    assert np.max(mix["relres"]) < 1e-4
    r = [c["restarts"] for c in mix["counters"]]
    if nstep < 20:
        assert min(r) >= 2 and len(set(r)) > 1, r
    ctx.close()


@pytest.mark.parametrize("nwant,nstep", [(8, 12), (5, 7)])
def test_es_maxit_allows_what_equal_restarts_would_take(nwant, nstep):
    """A mixed solve gets by with the es_maxit that the FP64 solve, whose restarts all keep nwant vectors, needs."""
    _, ctx = _ctx()
    kw = dict(nwant=nwant, nstep=nstep, es_tol=1e-10, ls_tol=1e-11)
    need = max(c["restarts"] for c in ctx.solve(KS, precision=fb.FP64, es_maxit=400, **kw)["counters"])
    out = ctx.solve(KS, precision=fb.MIXED, es_maxit=need, **kw)
    assert out["rc"] == fb.OK, [c["detail"] for c in out["counters"]]
    # and no more products than the cap stood for
    assert max(c["es_iter"] for c in out["counters"]) <= nstep + need * (nstep - nwant)
    ctx.close()
