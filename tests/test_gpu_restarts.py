"""Lanczos restarts: thick restarts in mixed precision (from a solve's second restart on), slots that restart
differently often in one batch, the restart product, es_maxit as a budget of products, and the memory a k-point takes."""
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


@pytest.mark.parametrize("nwant,nstep", [(1, 2), (3, 5), (30, 64), (48, 64)])
def test_restart_product_at_its_edges(nwant, nstep):
    """Row counts that leave every kind of remainder against the 32-row tiles (2 N = 1386 and, at Gamma, 1384), the
    smallest and the largest bases; random permittivities, so no bands coincide."""
    grid = (7, 9, 11)
    N = int(np.prod(grid))
    ctx = fb.Context(grid, np.full(3, 1.0 / 7), np.diag([n / 7 for n in grid]).reshape(-1), True)
    ctx.set_eps(np.random.default_rng(2).uniform(1.0, 13.0, 3 * N))
    k = np.array([[0.11, -0.23, 0.31], [0.0, 0.0, 0.0]])
    kw = dict(nwant=nwant, nstep=nstep, es_tol=1e-9, ls_tol=1e-11, es_maxit=1000)
    f64 = ctx.solve(k, precision=fb.FP64, **kw)
    mix = ctx.solve(k, precision=fb.MIXED, **kw)
    assert f64["rc"] == fb.OK and mix["rc"] == fb.OK
    assert min(c["restarts"] for c in f64["counters"] + mix["counters"]) >= 1
    assert np.max(np.abs(mix["freq"] - f64["freq"])) < 1e-7 * np.max(f64["freq"])
    assert max(np.max(f64["relres"]), np.max(mix["relres"])) < 1e-4
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


@pytest.mark.parametrize("general", [False, True])
def test_a_k_point_takes_no_more_memory_than_equal_restarts(general):
    """A slot's vectors fit what U with nstep + nwant + 2 columns and four FP64 and three FP32 CG vectors took."""
    n = 64
    if general:
        a = np.array([[1.0, 0, 0], [0, 1.0, 0], [0, -0.5, np.sqrt(0.75)]])
        grid = (n, n, n)
        h = np.diag(a) / n
        lat = dict(grid=grid, mesh_len=h, lattice_vec_a=a.reshape(-1), simple=False, m=(0, 0, int(0.5 / h[1] + 0.49), 0),
                   t1=(0.0, 1.0, 0.0))
    else:
        grid = (n, n, n)
        lat = dict(grid=grid, mesh_len=np.full(3, 1.0 / n), lattice_vec_a=np.eye(3).reshape(-1), simple=True)
    N, nwant, nstep, nb = n ** 3, 10, 40, 3
    M = 2 * N
    old = ((nstep + 1 + nwant + 1) * M + 4 * M + 3 * N + 2 * nwant * M + nwant * 3 * N + M) * 16 + 3 * M * 8 + 3 * N * 8
    B = np.random.default_rng(1).uniform(1.0, 13.0, 3 * N)
    k = np.array([[0.1, 0.2, 0.3], [0.11, 0.2, 0.3], [0.12, 0.2, 0.3]])
    kw = dict(nwant=nwant, nstep=nstep, es_tol=1e-2, ls_tol=1e-2, batch=nb)

    def run():
        ctx = fb.Context(**lat)
        ctx.set_eps(B)
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        ctx.solve(k, precision=fb.MIXED, **kw)
        used = free0 - torch.cuda.mem_get_info()[0]
        ctx.close()
        return used

    run()  # code, graphs and the driver's own pools are loaded
    assert run() <= nb * old + (64 << 20), (nb * old) >> 20
