"""High permittivity contrast: accuracy and cost of the CG in A_r^-1.

The three-term recurrences of the CG kernels lose accuracy with the square of the contrast, the
textbook form (the oracle's) with the contrast itself, so beyond a contrast of 32 the library restarts them
from the true residual.

  - FP64 A_r^-1: the true residual ||b - A x|| is at most ls_tol, or the oracle CG's where rounding does not
    let it reach ls_tol either (10% for the residual's own evaluation);
  - mixed precision: as many products per A_r^-1 as the form with search directions needs, 1.3 to 1.7 times those
    of an FP64 CG to 1e-10 at these contrasts (restated on the CPU in FP32 on these crystals; the
    three-term form with the default inner tolerance takes 1.9 to 3.4 times)."""
import numpy as np
import pytest

import fame_b200 as fb
import fame_oracle as fo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GEN, NEAR = (0.21, -0.13, 0.37), (2e-3, -1e-3, 1e-3)


def _par(n):
    return dict(grid=(n, n, n), N=n ** 3, mesh_len=np.full(3, 1.0 / n), lattice_vec_a=np.eye(3).reshape(-1), simple=True,
                m=(0, 0, 0, 0), t1=np.zeros(3))


def _eps(n, contrast, inverted):
    g = (np.arange(n) + 0.5) / n - 0.5
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    inside = (x * x + y * y + z * z < 0.09).reshape(-1)
    return np.tile(np.where(inside != inverted, float(contrast), 1.0), 3)


def _ctx(n, B):
    ctx = fb.Context.from_par(_par(n))
    ctx.set_eps(B)
    return ctx


@pytest.mark.parametrize("inverted", [False, True])
@pytest.mark.parametrize("contrast", [20, 100, 1e3, 1e4, 1e5])
@pytest.mark.parametrize("k", [GEN, NEAR], ids=["general", "near"])
def test_fp64_inverse_reaches_the_plain_form_s_residual(k, contrast, inverted):
    n = 14
    B = _eps(n, contrast, inverted)
    k = np.array(k)
    L = fo.lambdas(k, _par(n))
    s = np.concatenate([L.Lq_sqrt, L.Lq_sqrt])
    rng = np.random.default_rng(5)
    b = rng.standard_normal(2 * L.Nd) + 1j * rng.standard_normal(2 * L.Nd)
    b /= np.linalg.norm(b)
    ctx = _ctx(n, B)
    for tol in (1e-10, 1e-12, 1e-14):
        ref, _ = fo.cg(lambda p: fo.QBQ(p, L, 1.0 / B), b, tol, 2000)
        plain = np.linalg.norm(b - fo.QBQ(ref, L, 1.0 / B))
        y = torch.zeros(2 * L.Nd, dtype=torch.complex128, device="cuda")
        ctx.apply(fb.OP_INVAR, k, torch.from_numpy(b * s).to("cuda"), y, fb.FP64, fb.solver_params(ls_tol=tol, ls_maxit=2000))
        z = torch.from_numpy(y.cpu().numpy() * s).to("cuda")
        ctx.apply(fb.OP_QBQ, k, z, y, fb.FP64)  # each form's residual by its own operator: they differ by as much
        true = np.linalg.norm(b - y.cpu().numpy())
        assert true <= 1.1 * max(tol, plain), (tol, true, plain)
    ctx.close()


@pytest.mark.parametrize("inverted", [False, True])
@pytest.mark.parametrize("contrast,most", [(1e3, 1.75), (1e4, 2.0)])
def test_mixed_solve_takes_no_more_products(contrast, most, inverted):
    n = 14
    ctx = _ctx(n, _eps(n, contrast, inverted))
    k = np.array([GEN])
    kw = dict(nwant=4, nstep=24, es_tol=1e-10, ls_tol=1e-10)
    f64 = ctx.solve(k, precision=fb.FP64, **kw)
    f32 = ctx.solve(k, precision=fb.MIXED, **kw)
    assert f64["rc"] == fb.OK and f32["rc"] == fb.OK
    assert np.max(np.abs(f64["freq"] - f32["freq"])) < 1e-8 * np.max(f64["freq"])
    per = [o["counters"][0]["ls_iter"] / o["counters"][0]["es_iter"] for o in (f32, f64)]
    assert per[0] <= most * per[1], per
    ctx.close()


def test_permittivity_on_the_device_takes_the_same_path():
    n = 14
    B = _eps(n, 1e4, True)
    k = np.array([GEN])
    kw = dict(nwant=4, nstep=24, es_tol=1e-10, ls_tol=1e-10)
    a, b = _ctx(n, B), fb.Context.from_par(_par(n))
    b.set_eps_device(torch.from_numpy(B).to("cuda"))
    for prec in (fb.FP64, fb.MIXED):
        oa, ob = (c.solve(k, precision=prec, **kw) for c in (a, b))
        assert oa["counters"] == ob["counters"] and np.array_equal(oa["freq"], ob["freq"])
    # and back to an ordinary contrast: the counters of a context that never saw another
    low = _eps(n, 13, True)
    a.set_eps(low)
    c = _ctx(n, low)
    for prec in (fb.FP64, fb.MIXED):
        oa, oc = (q.solve(k, precision=prec, **kw) for q in (a, c))
        assert oa["counters"] == oc["counters"] and np.array_equal(oa["freq"], oc["freq"])
    for q in (a, b, c):
        q.close()


def test_fp64_solve_at_high_contrast_reports_a_cap():
    """ls_maxit bounds the products of an A_r^-1 solve, restarts included."""
    n = 14
    ctx = _ctx(n, _eps(n, 1e4, False))
    k = np.array([GEN])
    out = ctx.solve(k, nwant=4, nstep=20, es_maxit=1, es_tol=1e-10, ls_tol=1e-12, ls_maxit=20, precision=fb.FP64)
    c = out["counters"][0]
    assert out["rc"] == fb.ERR_NO_CONVERGENCE and c["detail"] & fb.KSTATUS_CG
    assert c["ls_iter"] <= 21 * c["es_iter"]  # the counter starts at 1 per solve
    ctx.close()
