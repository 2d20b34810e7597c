"""cg_coefficients (the scalars of the three-term CG recurrences) on the host: the textbook values on an ordinary
solve, and finite ones where the recurrence breaks down."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fame-isotropic-gpu_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include "fft_smem.cuh"
#include "state.cuh"
using namespace fame;
int main() {
  CgState st = {};
  double rAr, gm, rho;
  while (scanf("%d %lf %lf %lf %lf %lf", &st.iter, &st.r1, &st.r1p, &st.gm, &st.rho, &rAr) == 6) {
    cg_coefficients(st, rAr, gm, rho);
    printf("%.17g %.17g\n", gm, rho);
  }
}
"""


@pytest.fixture(scope="module")
def coefficients(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    d = tmp_path_factory.mktemp("coef")
    (d / "coef.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-arch=sm_100a", "--expt-relaxed-constexpr", "-I", CSRC, str(d / "coef.cu"), "-o",
                    str(d / "coef")], check=True)

    def run(rows):
        text = "\n".join(" ".join(repr(float(v)) if i else str(int(v)) for i, v in enumerate(r)) for r in rows)
        out = subprocess.run([str(d / "coef")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(float(v) for v in ln.split()) for ln in out.splitlines()]

    return run


def test_ordinary_solve(coefficients):
    """The scalars of CG on a diagonal matrix, step by step against gamma = rr / rAr and
    rho = 1 / (1 - gamma rr / (gamma_old rr_old rho_old)); the solve converges."""
    rng = np.random.default_rng(0)
    lam = rng.uniform(0.1, 1.0, 60)
    r, x = rng.standard_normal(60), np.zeros(60)
    b, ro, xo = r.copy(), np.zeros(60), np.zeros(60)
    rr0 = gm0 = 0.0
    rho0 = 1.0
    for k in range(1, 30):
        rr, rAr = r @ r, r @ (lam * r)
        gm, rho = coefficients([(k, rr, rr0, gm0, rho0, rAr)])[0]
        assert gm == rr / rAr
        assert rho == (1.0 if k == 1 else pytest.approx(1.0 / (1.0 - gm / gm0 * rr / rr0 / rho0), rel=1e-14))
        r, ro = rho * (r - gm * lam * r) + (1 - rho) * ro, r
        x, xo = rho * (x + gm * ro) + (1 - rho) * xo, x
        rr0, gm0, rho0 = rr, gm, rho
    assert np.linalg.norm(b - lam * x) < 1e-8 * np.linalg.norm(b)


def test_breakdown_gives_finite_coefficients(coefficients):
    nan, inf = float("nan"), float("inf")
    rows = [(5, 1e-4, 1e-3, 2.0, 1.5, 0.0),    # <r, A r> underflowed: no step
            (5, 1e-4, 1e-3, 2.0, 1.5, -1e-9),
            (5, 1e-4, 1e-3, 2.0, 1.5, nan),
            (6, 1e-4, 1e-4, 0.0, 1.0, 0.0),    # a second one in a row: 0 / 0
            (6, 1e-4, 1e-4, 0.0, 1.0, 1e-5),   # and a step after it
            (5, 2.0, 1.0, 1.0, 2.0, 2.0),      # denominator zero
            (5, 4.0, 1.0, 1.0, 1.0, 2.0),      # ... negative
            (5, 1.0, 1.0, 1.0, 1.0, 1.0 / (1.0 - 1e-15)),
            (5, inf, 1.0, 1.0, 1.0, 1.0),
            (5, 1.0, 1.0, 1.0, 1.0, 5e-324)]
    for row, (gm, rho) in zip(rows, coefficients(rows)):
        assert np.isfinite(gm) and gm >= 0, row
        assert np.isfinite(rho) and rho > 0, row
        if not row[5] > 0:
            assert gm == 0.0 and rho == 1.0, row
    assert coefficients([rows[4]])[0] == (10.0, 1.0)
