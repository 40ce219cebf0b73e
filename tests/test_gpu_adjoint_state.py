"""The handle's state after the adjoint's sweeps: ppf_adjoint_forward leaves u_{K-1} in the fields'
old_1 vectors and u_K in the current ones, as a run of K steps does, so that a block evaluated
afterwards gives u_K again; the backward sweep and the tangent model leave both as they were."""
import numpy as np
import pytest

from phasefield_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def states(steps):
    wl = W.coupled_acch_2d(refine=3, degree=2, size=32.0, dt=1e-3, n_precip=3)
    p = wl.make_problem()
    p.solve(steps)
    out = [p.download(f, age=1) for f in (0, 1)] if steps else [wl.initial[f] for f in (0, 1)]
    p.close()
    return out


def same(got, ref):
    for f in (0, 1):  # the same steps, up to the order of the scatter's FP64 additions
        assert np.linalg.norm(got[f] - ref[f]) <= 1e-13 * np.linalg.norm(ref[f]), f


@pytest.mark.parametrize("steps,slots", [(1, 1), (1, 3), (2, 1), (7, 1), (7, 3), (7, 8)])
def test_ages_after_the_sweeps(gpu_lib, steps, slots):
    p = W.coupled_acch_2d(refine=3, degree=2, size=32.0, dt=1e-3, n_precip=3).make_problem()
    before, last = states(steps - 1), states(steps)
    p.adjoint_forward(0, steps, slots)
    get = lambda age: [p.download(f, age=age) for f in (0, 1)]
    same(get(1), before)
    same(get(0), last)
    p.adjoint_backward(np.ones(2 * p.n_nodes))
    same(get(1), before)
    same(get(0), last)
    p.tangent_linear(0, 3, np.ones(2 * p.n_nodes), np.array([0.1, 0.2]))
    same(get(1), before)
    same(get(0), last)
    p.solve_block(0)
    same(get(0), last)
    p.close()
