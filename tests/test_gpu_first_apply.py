"""The first apply of a context reads no state that a solve would have set."""
import numpy as np
import pytest

import fame_b200 as fb
import fame_oracle as fo

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_first_apply_of_a_context_reads_no_stale_marker():
    """On 96^3 the plane kernels skip their work behind a fault marker; a new context's is clear whatever its memory
    held before."""
    n = 96
    N = n ** 3
    par = dict(grid=(n, n, n), N=N, mesh_len=np.full(3, 1.0 / n), lattice_vec_a=np.eye(3).reshape(-1), simple=True,
               m=(0, 0, 0, 0), t1=np.zeros(3))
    k = np.array([0.21, -0.13, 0.37])
    x = torch.randn(2 * N, dtype=torch.complex64, device="cuda")
    ref = fo.Qr(x.cpu().numpy().astype(np.complex128), fo.lambdas(k, par))
    for _ in range(3):
        ctx = fb.Context.from_par(par)
        # memory that held ones goes back to the driver just before the context allocates its workspace
        junk = [torch.full((1 << s,), 0x01010101, dtype=torch.int32, device="cuda") for s in (7, 10, 14, 18, 20, 22, 24, 26) for _ in range(4)]
        torch.cuda.synchronize()
        del junk
        torch.cuda.empty_cache()
        y = torch.zeros(3 * N, dtype=torch.complex64, device="cuda")
        ctx.apply(fb.OP_QR, k, x, y, fb.MIXED)
        assert np.linalg.norm(y.cpu().numpy() - ref) < 1e-5 * np.linalg.norm(ref)
        ctx.close()
