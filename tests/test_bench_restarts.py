"""bench.solve_bytes: the Lanczos steps and restart products of thick restarts, on a hand-computed case (N = 10, so
M = 20; nwant 2 of nstep 12: the first restart keeps 2 vectors, the others of a mixed solve 8)."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_thick_restarts_are_counted_as_they_run():
    c = dict(ls_iter=0, refine=0, es_iter=12 + 10 + 4 + 2, restarts=3)
    cols = sum(range(1, 13)) + sum(range(3, 13)) + sum(range(9, 13)) + 9 + 10  # j + 1 of every step
    column = 20 * 16
    want = (28 * 4 + 2 * cols + (13 + 3) + 2 * (13 + 9)) * column + 2 * 80 * 16
    assert bench.solve_bytes([c], 10, 2, 12, True) == want
    # FP64 restarts all keep nwant
    c64 = dict(ls_iter=0, refine=0, es_iter=12 + 10 + 6, restarts=2)
    cols = sum(range(1, 13)) + sum(range(3, 13)) + sum(range(3, 9))
    assert bench.solve_bytes([c64], 10, 2, 12, False) == (28 * 4 + 2 * cols + 2 * (13 + 3)) * column + 2 * 80 * 16


def test_cg_iteration_counts_the_form_that_runs():
    # N = 10: field 6 x 10 x 8, 1/eps 3 x 10 x 4, six vectors of 20 complex values
    assert bench.cg_iter_bytes(10) == 480 + 120 + 960
