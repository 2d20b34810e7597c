"""A mixed solve whose FP32 operator leaves the range of its numbers reports its A_r^-1 solves as not converged:
where 1/eps is infinite the first product is no number, where it is zero the CG finds no step (<r, A r> = 0)
and has to stay clear of 0 / 0."""
import numpy as np
import pytest

import fame_b200 as fb
from fixtures import load_pre

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-42, 1e46])
def test_fp32_operator_out_of_range_is_reported(eps):
    par = load_pre("sc16")
    ctx = fb.Context.from_par(par)
    ctx.set_eps(np.full(3 * int(np.prod(par["grid"])), eps))
    out = ctx.solve(np.array([[0.1, 0.2, 0.3]]), nwant=4, nstep=12, es_maxit=1, es_tol=1e-8, ls_tol=1e-8, inner_maxit=5,
                    precision=fb.MIXED)
    assert out["rc"] == fb.ERR_NO_CONVERGENCE
    assert out["counters"][0]["detail"] & fb.KSTATUS_CG
    # the context is usable afterwards
    ctx.set_material(par["binout"], par["material_num"], par["eps_in"], par["eps_out"])
    assert ctx.solve(par["kpoints"][1:2], nwant=4, nstep=20, es_tol=1e-8, ls_tol=1e-8, precision=fb.MIXED)["rc"] == fb.OK
    ctx.close()
