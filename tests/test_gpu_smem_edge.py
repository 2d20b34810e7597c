"""Grids whose stages take just under 48 KB of dynamic shared memory: with the kernels' static shared memory they
need the opt-in for more.  Operators against the oracle (FP64 1e-12, FP32 1e-5 relative, as on every grid), and
mixed against FP64 frequencies within the solves' own tolerance, 1e-10 on eigenvalues of A_r^-1 below 1, with
a factor of 100 for the largest of the bands."""
import numpy as np
import pytest

import fame_b200 as fb
import fame_oracle as fo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# plane FP64 47,456 bytes; pencil FP64 48,400 and FP32 47,432; plane FP32 47,400
GRIDS = [((53, 52, 6), "plane64"), ((10, 9, 121), "pencil"), ((75, 75, 4), "plane32")]


@pytest.mark.parametrize("grid,what", GRIDS)
def test_stages_just_under_48_kb(grid, what):
    nx, ny, nz = grid
    plane = ny * (nx | 1) + 2 * nx + 2 * ny
    size = {"plane64": 16 * plane, "plane32": 8 * plane, "pencil": 400 * nz}[what]
    assert 47000 < size <= 49152
    N = nx * ny * nz
    par = dict(grid=grid, N=N, mesh_len=np.full(3, 1.0 / nx), lattice_vec_a=np.diag([n / nx for n in grid]).reshape(-1),
               simple=True, m=(0, 0, 0, 0), t1=np.zeros(3))
    k = np.linalg.solve(par["lattice_vec_a"].reshape(3, 3), np.array([0.21, -0.13, 0.37]))
    rng = np.random.default_rng(N)
    B = rng.uniform(1.0, 13.0, 3 * N)
    ctx = fb.Context.from_par(par)
    ctx.set_eps(B)
    L = fo.lambdas(k, par)
    x = rng.standard_normal(2 * N) + 1j * rng.standard_normal(2 * N)
    v = rng.standard_normal(3 * N) + 1j * rng.standard_normal(3 * N)
    for prec, dt, tol in ((fb.FP64, torch.complex128, 1e-12), (fb.MIXED, torch.complex64, 1e-5)):
        for op, inp, ref in ((fb.OP_QR, x, fo.Qr(x, L)), (fb.OP_QRS, v, fo.Qrs(v, L)), (fb.OP_QBQ, x, fo.QBQ(x, L, 1.0 / B))):
            y = torch.zeros(ref.size, dtype=dt, device="cuda")
            ctx.apply(op, k, torch.from_numpy(inp).to("cuda", dt), y, prec)
            assert np.linalg.norm(y.cpu().numpy() - ref) < tol * np.linalg.norm(ref), (op, prec)
    kw = dict(nwant=3, nstep=24, es_tol=1e-10, ls_tol=1e-10)
    f64 = ctx.solve(k.reshape(1, 3), precision=fb.FP64, **kw)
    mix = ctx.solve(k.reshape(1, 3), precision=fb.MIXED, **kw)
    assert f64["rc"] == fb.OK and mix["rc"] == fb.OK
    assert np.max(np.abs(mix["freq"] - f64["freq"])) < 1e-8 * np.max(f64["freq"])
    ctx.close()
