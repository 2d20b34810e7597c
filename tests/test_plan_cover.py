"""The thread counts the host picks for the stage kernels cover every line of every FFT pass.

A host program built from the library's own headers walks grids with long and prime axes and prints,
for each stage, the threads of the launch rule (several launch sizes) and of the smallest plane-thread
option; here each pass is counted again: a butterfly pass of radix r stages T * max(1, E / r) of the
n / r butterflies of a line, a prime pass needs n / r * ceil(((r - 1) / 2 + 1) / MU) threads, and the
output-stationary pass that replaces it stages T * E of the n outputs."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fame-isotropic-gpu_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <initializer_list>
#include "fft_smem.cuh"
#include "geom_policy.cuh"
#include "geometry.h"
using namespace fame;
static void axis(const char* what, int real, int T, int emax, int mu, const AxisPlan& p) {
  printf("%s %d %d %d %d %d", what, real, T, emax, mu, p.n);
  for (int i = 0; i < p.npass; i++) printf(" %d", p.radix[i]);
  printf("\n");
}
template <typename R> static void grid(const Geom& g) {
  const int lp = plane_level(g), ls = pencil_level(g);
  for (long slots : {1L, 4L, 20L, 64L}) {
    for (int T : {plane_threads_rule<R>(g, lp, slots * g.Ls), std::max(64, plane_threads_min<R>(g))})
      for (const AxisPlan* p : {&g.pf, &g.pm}) axis("plane", sizeof(R), T, Emax<R>::v, PrimeBlock<R, false>::mu, *p);
    axis("pencil", sizeof(R), pencil_threads_rule<R>(g, ls, slots), Emax<R>::v, PrimeBlock<R, true>::mu, g.ps);
  }
}
int main() {
  int nx, ny, nz;
  while (scanf("%d %d %d", &nx, &ny, &nz) == 3) {
    fame_lattice L = {};
    L.grid[0] = nx, L.grid[1] = ny, L.grid[2] = nz;
    for (double& h : L.mesh_len) h = 0.1;
    L.simple = 1;
    for (int order = 0; order < kNumRadixOrders; order++) {
      Geom g;
      std::string err;
      if (layout_geom(L, g, 1L << 28, err, order) != FAME_OK) continue;
      grid<double>(g);
      grid<float>(g);
    }
  }
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    d = tmp_path_factory.mktemp("plans")
    (d / "plans.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-arch=sm_100a", "--expt-relaxed-constexpr", "-I", CSRC, str(d / "plans.cu"),
                    "-o", str(d / "plans")], check=True)
    grids = [(n, 2, m) for n in range(17, 2400, 7) for m in (2, 250)]  # long fast axes, 2 mod cross-sections
    grids += [(521, 2, 250), (2, 521, 250), (1042, 2, 30), (577, 3, 40), (4, 3, 577), (2, 2, 581), (2048, 3, 6), (107, 92, 128)]
    text = "\n".join("%d %d %d" % g for g in grids)
    out = subprocess.run([str(d / "plans")], input=text, capture_output=True, text=True, check=True).stdout
    return [(ln.split()[0], [int(v) for v in ln.split()[1:]]) for ln in out.splitlines()]


def test_every_pass_covers_whole_lines(plans):
    assert len(plans) > 10000
    bad = set()
    for what, (real, T, emax, mu, n, *radices) in plans:
        for r in radices:
            nb = n // r
            if r > 13:
                cells = nb * (((r - 1) // 2 + mu) // mu)
                ok = cells <= T or T * emax >= n
            else:
                ok = T * max(1, emax // r) >= nb
            if not ok:
                bad.add((what, real, T, n, r))
    assert not bad, sorted(bad)[:20]


def test_prime_pass_runs_where_a_block_can_hold_it(plans):
    """The output-stationary pass takes r loads per output; it is only for lines whose cells exceed a CTA."""
    for what, (real, T, emax, mu, n, *radices) in plans:
        for r in radices:
            cells = n // r * (((r - 1) // 2 + mu) // mu)
            if r > 13 and cells <= (512 if what == "plane" else 256):
                assert cells <= T, (what, real, T, n, r)
