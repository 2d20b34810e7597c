"""Operators on grids with one long axis and a thin cross-section: the plane CTAs are small there, and
a prime factor of the axis needs more of their threads than the rule for launch sizes asks for.

Against the oracle, FP64 within 1e-12 relative and FP32 within 1e-5: the longest sum is 577 terms, whose
rounding (sqrt(577) units of 2^-53 and 2^-24 at most in the mean) leaves two orders to spare."""
import numpy as np
import pytest

import fame_b200 as fb
import fame_oracle as fo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# (grid, plane-thread option): 521 = a prime axis of 131 FP64 cells; 1042 = 2 x 521; 255 = 15 x 17
GRIDS = [((521, 2, 250), 0), ((2, 521, 60), 0), ((1042, 2, 6), 0), ((255, 3, 8), 0), ((521, 2, 6), 64), ((3, 577, 4), 64),
         ((4, 3, 577), 0)]


@pytest.mark.parametrize("grid,threads", GRIDS)
def test_operators_on_long_axes(grid, threads):
    N = int(np.prod(grid))
    par = dict(grid=grid, N=N, mesh_len=np.full(3, 1.0 / grid[0]), lattice_vec_a=np.diag([n / grid[0] for n in grid]).reshape(-1),
               simple=True, m=(0, 0, 0, 0), t1=np.zeros(3))
    k = np.linalg.solve(par["lattice_vec_a"].reshape(3, 3), np.array([0.21, -0.13, 0.37]))
    rng = np.random.default_rng(N)
    B = rng.uniform(1.0, 13.0, 3 * N)
    ctx = fb.Context.from_par(par)
    ctx.set_option("plane_threads64", threads)
    ctx.set_option("plane_threads32", threads)
    ctx.set_eps(B)
    L = fo.lambdas(k, par)
    x = rng.standard_normal(2 * N) + 1j * rng.standard_normal(2 * N)
    v = rng.standard_normal(3 * N) + 1j * rng.standard_normal(3 * N)
    for prec, dt, tol in ((fb.FP64, torch.complex128, 1e-12), (fb.MIXED, torch.complex64, 1e-5)):
        for op, inp, ref in ((fb.OP_QR, x, fo.Qr(x, L)), (fb.OP_QRS, v, fo.Qrs(v, L)), (fb.OP_QBQ, x, fo.QBQ(x, L, 1.0 / B))):
            y = torch.zeros(ref.size, dtype=dt, device="cuda")
            ctx.apply(op, k, torch.from_numpy(inp).to("cuda", dt), y, prec)
            got = y.cpu().numpy().astype(np.complex128)
            assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref), (op, prec)
    ctx.close()
