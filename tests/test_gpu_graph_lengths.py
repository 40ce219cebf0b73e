"""Increment graphs over a handle's life: what a run replays does not depend on the length of the runs
before it, and runs continue each other exactly. The state after each run against plain launches within
1e-12 relative L2 (the order of the scatter's FP64 additions)."""
import ctypes as C

import numpy as np
import pytest

from phasefield_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def plain_cell_launches(p, n):
    """Cell launches of n further increments that no graph replayed."""
    p._check(p.lib.ppf_kernel_stats_reset(p.h))
    p.solve(p.get_time()[0] + n - 1)
    cells = C.c_longlong()
    p._check(p.lib.ppf_kernel_stats(p.h, None, C.byref(cells), None))
    return cells.value


@pytest.mark.parametrize("first", [3, 10, 17, 100, 400])
def test_replays_do_not_depend_on_the_first_run(gpu_lib, first):
    wl = W.coupled_acch_2d(refine=3, degree=1, size=32.0, dt=1e-4, n_precip=3)  # one block, periods of 2
    p = wl.make_problem()
    p.solve(1)
    plain_cell_launches(p, first)
    for n in (10, 17, 3, 100, 10, 17, 3, 100, 400, 3, 10, 17, 100):
        plain_cell_launches(p, n)  # both phases, short and long graphs
    for n in (3, 10, 17, 2, 100, 1, 100, 17, 10, 3):
        assert plain_cell_launches(p, n) == n % 2, n
    p.close()


@pytest.mark.parametrize("runs", [(4, 6, 6), (100, 10, 17, 10, 100), (3, 3, 3, 40, 150, 7), (150, 16, 150, 2), (17, 17, 17, 17)])
def test_runs_continue_each_other(gpu_lib, runs):
    """Graphs replayed in a later run, at both phases of the rotation, after calls that leave the fields on
    their other accumulators (an odd number of products) and after staged uploads of the state."""
    wl = W.coupled_acch_2d(refine=3, degree=2, size=32.0, dt=1e-4, n_precip=3)
    for between in ("nothing", "products", "uploads"):
        res = []
        for use_graph in (0, 1):
            p = wl.make_problem()
            p._check(p.lib.ppf_set_use_graph(p.h, use_graph))
            p.solve(1)
            keep, out = [], []
            for i, n in enumerate(runs):
                p.solve(1 + sum(runs[:i + 1]))
                out += [p.download_solution(f) for f in (0, 1)]
                if between == "products":
                    for _ in range(1 + i % 2 * 2):
                        p.apply(0, 0, None, scale=1)
                if between == "uploads":
                    for f in (0, 1):
                        keep.append(0.999 * p.download(f, age=1))
                        p._check(p.lib.ppf_upload_state_staged(p.h, f, 1, keep[-1].ctypes.data_as(C.POINTER(C.c_double))))
            assert p.get_time()[0] == 2 + sum(runs)
            p._check(p.lib.ppf_wait(p.h))
            res.append(out)
            p.close()
        for a, b in zip(*res):
            assert rel_l2(b, a) < 1e-12, between
