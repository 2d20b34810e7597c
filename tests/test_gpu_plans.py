"""Runtime FFT plans, pencil tiles and the CG kernels at the edges of their ranges.

Grids whose axes take every butterfly radix 2..13 (alone and as a second pass with Stockham
twiddles), three-pass axes, prime factors >= 17, planes whose size leaves every remainder against
the 16- and 32-position pencil tiles and the 16-byte copies (odd, 2 mod 4, 0 mod 4), and the
smallest grids.  Operators against the oracle: FP64 within 1e-12 relative (about 100 roundings of
2^-53 in a chain of log2(N) butterflies leave two orders to spare), FP32 within 1e-5; A_r^-1 with
its CG stopped at 1e-12 within 1e-9 (residual over the smallest eigenvalue)."""
import numpy as np
import pytest

import fame_b200 as fb
import fame_oracle as fo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (grid, general lattice, wave vector is Gamma)
GRIDS = [((2, 2, 2), False, False), ((3, 2, 5), False, True), ((13, 11, 9), False, False), ((12, 10, 6), False, True),
         ((7, 8, 4), False, False), ((49, 22, 15), False, False), ((20, 26, 27), False, False),
         ((33, 36, 10), False, False), ((75, 35, 6), False, False), ((40, 39, 50), False, True),
         ((34, 19, 51), False, False), ((9, 10, 12), True, False), ((26, 21, 18), True, True), ((46, 22, 17), True, False)]


def _par(grid, general):
    if not general:
        return dict(grid=grid, N=int(np.prod(grid)), mesh_len=np.full(3, 1.0 / grid[0]),
                    lattice_vec_a=np.diag([n / grid[0] for n in grid]).reshape(-1), simple=True, m=(0, 0, 0, 0),
                    t1=np.zeros(3))
    a = np.array([[1.2, 0, 0], [0, 1.0, 0], [0, -0.5, np.sqrt(0.75)]])  # hexagonal
    h = np.diag(a) / np.array(grid)
    return dict(grid=grid, N=int(np.prod(grid)), mesh_len=h, lattice_vec_a=a.reshape(-1), simple=False,
                m=(0, 0, int(0.5 / h[1] + 0.49), 0), t1=np.array([0.0, 1.0, 0.0]))


def _rel(y, ref):
    return np.linalg.norm(y.cpu().numpy().astype(np.complex128) - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("grid,general,gamma", GRIDS)
def test_operators_and_cg_at_plan_edges(grid, general, gamma):
    par = _par(grid, general)
    N = par["N"]
    a = par["lattice_vec_a"].reshape(3, 3)
    k = np.zeros(3) if gamma else np.linalg.solve(a, np.array([0.21, -0.13, 0.37]))
    rng = np.random.default_rng(N)
    B = rng.uniform(1.0, 13.0, 3 * N)
    ctx = fb.Context.from_par(par)
    ctx.set_eps(B)
    L = fo.lambdas(k, par)
    x = rng.standard_normal(2 * L.Nd) + 1j * rng.standard_normal(2 * L.Nd)
    v = rng.standard_normal(3 * N) + 1j * rng.standard_normal(3 * N)
    for prec, dt, tol in ((fb.FP64, torch.complex128, 1e-12), (fb.MIXED, torch.complex64, 1e-5)):
        for op, inp, ref in ((fb.OP_QR, x, fo.Qr(x, L)), (fb.OP_QRS, v, fo.Qrs(v, L)),
                             (fb.OP_QBQ, x, fo.QBQ(x, L, 1.0 / B))):
            y = torch.zeros(ref.size, dtype=dt, device="cuda")
            ctx.apply(op, k, torch.from_numpy(inp).to("cuda", dt), y, prec)
            assert _rel(y, ref) < tol, (op, prec)
    y = torch.zeros(2 * L.Nd, dtype=torch.complex128, device="cuda")
    ctx.apply(fb.OP_INVAR, k, torch.from_numpy(x).to("cuda"), y, fb.FP64, fb.solver_params(ls_tol=1e-12, ls_maxit=1000))
    assert _rel(y, fo.invAr(x, L, 1.0 / B, 1e-12, 1000)) < 1e-9
    if N > 100:  # mixed precision (FP32 CG under FP64 refinement) against FP64
        kw = dict(nwant=3, nstep=16, es_tol=1e-10, ls_tol=1e-10)
        f64 = ctx.solve(k, precision=fb.FP64, **kw)
        f32 = ctx.solve(k, precision=fb.MIXED, **kw)
        assert f64["rc"] == fb.OK and f32["rc"] == fb.OK
        assert np.max(np.abs(f64["freq"] - f32["freq"])) < 1e-6 * np.max(f64["freq"])
    ctx.close()


@pytest.mark.parametrize("gamma", [False, True])
def test_fp64_half_planes(gamma):
    """The 96^3 FP64 plane stages share a component's plane between two CTAs."""
    par = _par((96, 96, 96), False)
    N = par["N"]
    k = np.zeros(3) if gamma else np.array([0.21, -0.13, 0.37])
    rng = np.random.default_rng(N)
    B = rng.uniform(1.0, 13.0, 3 * N)
    ctx = fb.Context.from_par(par)
    ctx.set_eps(B)
    L = fo.lambdas(k, par)
    x = rng.standard_normal(2 * L.Nd) + 1j * rng.standard_normal(2 * L.Nd)
    v = rng.standard_normal(3 * N) + 1j * rng.standard_normal(3 * N)
    for op, inp, ref in ((fb.OP_QR, x, fo.Qr(x, L)), (fb.OP_QRS, v, fo.Qrs(v, L)), (fb.OP_QBQ, x, fo.QBQ(x, L, 1.0 / B))):
        y = torch.zeros(ref.size, dtype=torch.complex128, device="cuda")
        ctx.apply(op, k, torch.from_numpy(inp).to("cuda"), y, fb.FP64)
        assert _rel(y, ref) < 1e-12, op
    ctx.close()
