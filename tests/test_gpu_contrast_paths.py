"""The FP64 restarts from the true residual (permittivity contrast beyond 32) on every form of the operator stages:
general lattices with runtime and static plans, the 96^3 half planes, several k-points with different counts in one
batch, the Gamma point, the host-driven loops, and a loop cap.

Residuals by the library's own operator, at most ls_tol or 8 contrast 2^-53 of the right-hand side (what the
library accepts as rounding).  Frequencies: FP64 against mixed precision, 1e-8 of the largest (es_tol 1e-10)."""
import numpy as np
import pytest

import fame_b200 as fb
from fixtures import load_pre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _sphere(N, grid, contrast):
    g = [(np.arange(n) + 0.5) / n - 0.5 for n in grid]
    z, y, x = np.meshgrid(g[2], g[1], g[0], indexing="ij")
    return np.tile(np.where((x * x + y * y + z * z < 0.09).reshape(-1), float(contrast), 1.0), 3)


def _lattice(name):
    if name == "simple96":
        return dict(grid=(96, 96, 96), mesh_len=np.full(3, 1 / 96), lattice_vec_a=np.eye(3).reshape(-1), simple=True)
    if name in ("fcc64", "hex36"):
        r2, r3, r6 = np.sqrt([2.0, 3.0, 6.0])
        if name == "fcc64":
            a, grid, t1 = np.array([[1 / r2, 0, 0], [0.5 / r2, r6 / 4, 0], [0.5 / r2, r6 / 12, 1 / r3]]), (64, 55, 52), np.zeros(3)
        else:
            a, grid, t1 = np.array([[1.2, 0, 0], [0, 1.0, 0], [0, -0.5, r3 / 2]]), (36, 30, 26), np.array([0.0, 1.0, 0.0])
        h = np.array([a[i, i] / grid[i] for i in range(3)])
        b1 = a[1, 0] + (a[0, 0] if a[1, 0] < 0 else 0.0)
        a3 = a[2] + t1
        m = (int(round(b1 / h[0])), int(round(a3[0] / h[0])), int(a3[1] / h[1] + 0.49), 0)
        return dict(grid=grid, mesh_len=h, lattice_vec_a=a.reshape(-1), simple=False, m=m, t1=t1)
    p = load_pre(name)
    return dict(grid=p["grid"], mesh_len=p["mesh_len"], lattice_vec_a=p["lattice_vec_a"], simple=p["simple"], m=p["m"], t1=p["t1"])


@pytest.mark.parametrize("name", ["fcc16", "bcc12", "hex12", "hex36", "fcc64", "simple96"])
@pytest.mark.parametrize("contrast", [40, 1e4])
@pytest.mark.parametrize("k", [(0.21, -0.13, 0.37), (0.0, 0.0, 0.0)], ids=["general", "gamma"])
def test_inverse_reaches_ls_tol(name, contrast, k):
    lat = _lattice(name)
    N = int(np.prod(lat["grid"]))
    ctx = fb.Context(**lat)
    ctx.set_eps(_sphere(N, lat["grid"], contrast))
    k = np.array(k)
    n = 2 * fb.reduced_size(ctx._lat, k)
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.view_as_complex(torch.randn(n, 2, dtype=torch.float64, device="cuda", generator=gen))
    x /= torch.linalg.vector_norm(x)
    # sqrt(Lambda): A_r^-1 x = (1/s) QBQ^-1 (1/s) x; s^-2 x is A_r^-1 x in a homogeneous medium
    one = fb.Context(**lat)
    one.set_eps(np.ones(3 * N))
    s2 = torch.empty_like(x)
    one.apply(fb.OP_INVAR, k, torch.ones_like(x), s2, fb.FP64, fb.solver_params(ls_tol=1e-15, ls_maxit=50))
    s = torch.rsqrt(s2.real)
    one.close()
    b = x / s
    for tol in (1e-10, 1e-12):
        y = torch.empty_like(x)
        ctx.apply(fb.OP_INVAR, k, x, y, fb.FP64, fb.solver_params(ls_tol=tol, ls_maxit=2000))
        q = torch.empty_like(x)
        ctx.apply(fb.OP_QBQ, k, y * s, q, fb.FP64)
        nb = float(torch.linalg.vector_norm(b))
        true = float(torch.linalg.vector_norm(b - q))
        assert true <= max(1.1 * tol, 8 * 2.0 ** np.ceil(np.log2(contrast)) * 2.0 ** -53 * nb), (tol, true, nb)
    ctx.close()


@pytest.mark.parametrize("name", ["fcc16", "sc16"])
def test_batches_graphs_and_host_loops_agree(name):
    lat = _lattice(name)
    N = int(np.prod(lat["grid"]))
    ctx = fb.Context(**lat)
    ctx.set_eps(_sphere(N, lat["grid"], 3e3))
    k = np.array([[0.21, -0.13, 0.37], [0.02, 0.01, -0.015], [0.31, 0.11, -0.22]])
    kw = dict(nwant=4, nstep=24, es_tol=1e-10, ls_tol=1e-11)
    a = ctx.solve(k, precision=fb.FP64, batch=3, **kw)
    b = ctx.solve(k, precision=fb.FP64, batch=3, use_graph=0, **kw)
    c = ctx.solve(k, precision=fb.FP64, batch=1, **kw)
    m = ctx.solve(k, precision=fb.MIXED, batch=3, **kw)
    assert all(o["rc"] == fb.OK for o in (a, b, c, m))
    assert np.array_equal(a["freq"], b["freq"]) and a["counters"] == b["counters"]
    assert all(q["refine"] >= q["es_iter"] for q in a["counters"])
    for o in (c, m):
        assert np.max(np.abs(o["freq"] - a["freq"])) < 1e-8 * np.max(a["freq"])
    # a cap on the loops ends the solve with a status, and the context goes on
    ctx.set_loop_cap(2)
    with pytest.raises(fb.FameError) as e:
        ctx.solve(k, precision=fb.FP64, batch=3, **kw)
    assert e.value.code == fb.ERR_WATCHDOG
    ctx.set_loop_cap(0)
    d = ctx.solve(k, precision=fb.FP64, batch=3, **kw)
    assert d["rc"] == fb.OK and np.array_equal(a["freq"], d["freq"])
    ctx.close()
