"""A plan cache line of another version of the plans is not applied: its radix orders and thread counts name
other plans than the ones they were timed on."""
import pytest

import fame_b200 as fb
from fixtures import load_pre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_unversioned_cache_lines_are_ignored(tmp_path):
    par = load_pre("fcc16")
    ctx = fb.Context.from_par(par)
    ctx.set_material(par["binout"], par["material_num"], par["eps_in"], par["eps_out"])
    k = par["kpoints"][1]
    cache = tmp_path / "plans.txt"
    g = par["grid"]
    old = (f"grid={g[0]}x{g[1]}x{g[2]} general=1 precision=fp64 batch=1 | radix_order=2 plane_threads32=512 "
           "plane_threads64=512 prefetch=1\n")
    cache.write_text(old)
    assert "(cached)" not in ctx.tune(k, fb.FP64, batch=1, cache_file=str(cache))
    lines = cache.read_text().splitlines()
    assert lines[0] + "\n" == old and len(lines) == 2  # timed, and appended
    assert ctx.tune(k, fb.FP64, batch=1, cache_file=str(cache)).endswith("(cached)")
    ctx.close()
