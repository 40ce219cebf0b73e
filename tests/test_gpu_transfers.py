"""Multigrid transfers of degrees 3 and 4, which go axis by axis: GMG-CG against the oracle, in 2-D and
3-D, periodic and not, FP64 and with FP32 levels. Bars of tests/test_gpu_linear.py: iteration counts
within 10 % (1.5 times with FP32 levels), solutions within 1e-8 relative L2."""
import numpy as np
import pytest

from oracle import pyoracle as po
from phasefield_gb300 import workloads as W
from phasefield_gb300.problem import RectangularMesh

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# (smoother degrees with which the oracle's V-cycle contracts)
@pytest.mark.parametrize("dim,degree,sub,periodic,smoother", [
    (2, 3, (2, 2), (0, 0, 0), 6), (2, 4, (3, 3), (0, 1, 0), 10), (3, 3, (1, 1, 1), (0, 0, 0), 10),
    (3, 3, (1, 1, 1), (0, 1, 1), 6), (3, 4, (1, 1, 1), (0, 0, 1), 6),
])
def test_gmg_of_higher_degrees(gpu_lib, dim, degree, sub, periodic, smoother):
    wl = W.eshelby_3d(refine=0, degree=degree, size=16.0, n_incl=4, dim=dim)
    wl.mesh = RectangularMesh(dim=dim, degree=degree, size=(16.0,) * dim + (1.0,) * (3 - dim),
                              subdivisions=sub + (1,) * (3 - dim), global_refinement=2, periodic=periodic)
    prm = dict(tolerance_type=1, tolerance=1e-10, max_iterations=300, preconditioner=2, mg_depth=3, smoother_degree=smoother)
    o = po.Oracle(wl)
    o.set_linear_params(0, **prm)
    rc, oits, _ = o.linear_solve(0)
    assert rc == 0
    for mixed in (0, 1):
        p = wl.make_problem()
        p.set_linear_params(0, mixed_precision=mixed, **prm)
        its, res = p.linear_solve(0)
        assert res < 1e-10
        assert its <= (1.5 * oits + 2 if mixed else oits + max(2, 0.1 * oits))
        assert mixed or its >= oits - max(2, 0.1 * oits)
        assert rel_l2(p.download(0), o.get(0)) < 1e-8, mixed
        p.close()
