"""Set-up of a block's first solve while the default stream is busy: the solver's work space is zeroed
in the order of the handle's own stream, which does not wait for the default one. Solutions against
the oracle with the bars of tests/test_gpu_newton.py and tests/test_gpu_linear.py (1e-8)."""
import numpy as np
import pytest

from oracle import pyoracle as po
from phasefield_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def busy_default_stream():
    import torch
    with torch.cuda.stream(torch.cuda.default_stream()):
        torch.cuda._sleep(200_000_000)  # about a tenth of a second


@pytest.mark.parametrize("preconditioner", [0, 1])
def test_first_newton_solve(gpu_lib, preconditioner):
    import torch
    wl = W.allen_cahn_implicit_2d(refine=4, dt=1.0)
    lin = dict(tolerance_type=1, tolerance=1e-12, max_iterations=3000, preconditioner=preconditioner, smoother_degree=4)
    p, o = wl.make_problem(), po.Oracle(wl)
    for s in (p, o):
        s.set_linear_params(0, **lin)
        s.set_newton_params(0, max_iterations=50, tolerance=1e-10)
    p.solve(0)  # the initial state (no solve of the block yet)
    assert o.run(0) == 0
    torch.cuda.synchronize()
    busy_default_stream()
    its, _, res = p.newton_solve(0)
    rc, oits, _, _ = o.newton_solve(0)
    assert rc == 0 and its == oits and res < 1e-10
    assert rel_l2(p.download(0), o.get(0, 0)) < 1e-8


@pytest.mark.parametrize("preconditioner", [0, 1, 2])
def test_first_linear_solve(gpu_lib, preconditioner):
    import torch
    wl = W.eshelby_3d(refine=2, degree=2, size=16.0, n_incl=5)
    prm = dict(tolerance_type=1, tolerance=1e-10, max_iterations=1500, preconditioner=preconditioner, mg_depth=2,
               smoother_degree=4)
    p, o = wl.make_problem(), po.Oracle(wl)
    p.set_linear_params(0, **prm)
    o.set_linear_params(0, **prm)
    torch.cuda.synchronize()
    busy_default_stream()
    _, res = p.linear_solve(0)
    rc, _, _ = o.linear_solve(0)
    assert rc == 0 and res < 1e-10
    assert rel_l2(p.download(0), o.get(0)) < 1e-8
