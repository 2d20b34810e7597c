"""Calls on device tensors are ordered after the work that the caller has queued on its torch stream."""
import numpy as np
import pytest

import fame_b200 as fb
from fixtures import edge_eps, load_pre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BUSY = 100_000_000  # clock cycles of a kernel in front of the write: about 50 ms


def _ctx():
    par = load_pre("sc16")
    ctx = fb.Context.from_par(par)
    ctx.set_eps(edge_eps(par))
    return par, ctx


@pytest.mark.parametrize("side_stream", [False, True])
def test_apply_waits_for_the_input(side_stream):
    par, ctx = _ctx()
    k = np.array([0.1, 0.2, 0.3])
    N = int(np.prod(par["grid"]))
    src = torch.randn(2 * N, dtype=torch.complex128, device="cuda")
    want = torch.zeros_like(src)
    ctx.apply(fb.OP_QBQ, k, src, want, fb.FP64)
    x, y = torch.zeros_like(src), torch.zeros_like(src)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.current_stream()):
        torch.cuda._sleep(BUSY)
        x.copy_(src)
        ctx.apply(fb.OP_QBQ, k, x, y, fb.FP64)
        got = y.clone()
        torch.cuda.current_stream().synchronize()
    assert torch.equal(got, want)
    ctx.close()


def test_permittivity_and_gradient_wait_for_their_tensors():
    par, ctx = _ctx()
    k = np.array([[0.1, 0.2, 0.3]])
    N = int(np.prod(par["grid"]))
    B = torch.from_numpy(edge_eps(par)).to("cuda")
    kw = dict(nwant=4, nstep=20, es_tol=1e-10, ls_tol=1e-10)
    want = ctx.solve(k, **kw)["freq"]
    ctx.set_eps(np.full(3 * N, 2.0))
    late = torch.ones_like(B)
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    late.copy_(B)
    ctx.set_eps_device(late)
    out = ctx.solve(k, vectors_on_device=True, **kw)
    assert np.array_equal(out["freq"], want)
    g = np.ones(4)
    ref = ctx.adjoint_vjp(0, out["freq"][0], g).clone()
    buf = torch.empty(N, dtype=torch.float64, device="cuda")
    torch.cuda._sleep(BUSY)
    buf.zero_()  # queued before the call that fills it
    ctx.adjoint_vjp(0, out["freq"][0], g, out=buf)
    torch.cuda.synchronize()
    assert torch.equal(buf, ref)
    ctx.close()
