"""The lane kernel far from O(1) (include/prismspf/gpu/cell_kernel_lanes.cuh): a cell keeps the
accuracy of its own largest value down to 1e-288, against the oracle. One operator within
1e-12 relative L2 (the bar of tests/test_gpu_lane_kernel.py), steps within 1e-9."""
import numpy as np
import pytest

from oracle import pyoracle as po
from phasefield_gb300 import ensemble as E
from phasefield_gb300 import workloads as W
from phasefield_gb300.problem import RectangularMesh

pytestmark = pytest.mark.gpu


def rel_l2(a, b, scale=1.0):
    a, b = a / scale, b / scale  # (the squares of values this small underflow)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def elasticity(dim, degree, size):
    wl = W.eshelby_3d(refine=0, degree=degree, size=8.0, n_incl=1, dim=dim)
    sub = (5, 4, 3)[:dim] + (1,) * (3 - dim)
    wl.mesh = RectangularMesh(dim=dim, degree=degree, size=tuple(s * n for s, n in zip(size, sub)), subdivisions=sub)
    return wl


@pytest.mark.parametrize("scale", [1e-253, 1e-270, 1e-283])
@pytest.mark.parametrize("dim,degree,size,mode", [
    (2, 1, (2.0, 2.0, 1.0), 4), (2, 2, (1.0, 3.0, 1.0), 5), (3, 1, (1.3, 0.7, 2.1), 5), (3, 2, (1.7, 1.7, 1.7), 4),
])
def test_small_fields_several_components(gpu_lib, monkeypatch, dim, degree, size, mode, scale):
    monkeypatch.setenv("PPF_CONTRACTION_MODE", str(mode))
    wl = elasticity(dim, degree, size)
    p, o = wl.make_problem(), po.Oracle(wl)
    u = np.random.default_rng(6).normal(size=p.field_length(0))
    assert rel_l2(p.apply(0, 1, u * scale, scale=0), o.apply(0, 1, u * scale, scale=0), scale) < 1e-12
    assert p.contraction_mode(0, 1) == mode
    # small values in one half of the box next to O(1) values in the other
    x = W.lattice_coordinates(wl.mesh)[:, 0] / wl.mesh.size[0]
    s = np.tile(np.where(x < 0.45, scale, 1.0), dim)
    got, ref = p.apply(0, 1, u * s, scale=0), o.apply(0, 1, u * s, scale=0)
    far = np.tile(x < 0.15, dim)
    assert rel_l2(got, ref) < 1e-12 and rel_l2(got[far], ref[far], scale) < 1e-12


@pytest.mark.parametrize("scale", [1e-253, 1e-270, 1e-283])
@pytest.mark.parametrize("dim,degree,size,mode", [
    (2, 1, (8.0, 8.0, 1.0), 4), (2, 2, (8.0, 5.0, 1.0), 5), (3, 1, (8.0, 5.0, 3.0), 5), (3, 2, (7.0, 7.0, 7.0), 4),
])
def test_small_fields_one_component(gpu_lib, monkeypatch, dim, degree, size, mode, scale):
    """c zero (no value term) and mu small: the gradient terms alone."""
    monkeypatch.setenv("PPF_CONTRACTION_MODE", str(mode))
    wl = W.cahn_hilliard_3d(refine=0, degree=degree, dim=dim, size=1.0, subdivisions=(7, 7, 7)[:dim] + (1,) * (3 - dim),
                            dt=1e-3)
    wl.mesh.size = size
    p, o = wl.make_problem(), po.Oracle(wl)
    mu = np.random.default_rng(8).normal(size=p.n_nodes) * scale
    zero = np.zeros(p.n_nodes)
    for f, v, age in ((0, zero, 0), (0, zero, 1), (1, mu, 1)):
        p.upload(f, v, age=age)
        o.set(f, v, age=age)
    assert rel_l2(p.apply(0, 0, None, scale=1), o.apply(0, 0, None, scale=1), scale) < 1e-12
    assert p.contraction_mode(0, 0) == mode


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("scale", [1e-253, 1e-283])
def test_small_fields_in_an_ensemble(gpu_lib, degree, scale):
    sub = [(48, 64), (64, 50), (61, 47), (64, 64), (33, 70)]
    meshes = [RectangularMesh(dim=2, degree=degree, size=(2.0 * a, 2.0 * b, 1.0), subdivisions=(a, b, 1)) for a, b in sub]
    rng = np.random.default_rng(degree)
    ics = [rng.uniform(0.0, 1.0, size=int(np.prod(m.nodes))) * scale for m in meshes]
    ens = E.Ensemble(meshes, [1.0] * len(sub), [2.0] * len(sub), 0.01)
    for i, ic in enumerate(ics):
        ens.upload(i, ic)
    ens.run(3)
    for i, m in enumerate(meshes):
        wl = W.allen_cahn_2d(refine=0, degree=degree, m_well=1.0, kappa=2.0, dt=0.01, subdivisions=sub[i])
        wl.mesh, wl.initial = m, {0: ics[i]}
        o = po.Oracle(wl)
        assert o.run(3) == 0
        assert rel_l2(ens.download(i), o.get(0, 1), scale) < 1e-9, sub[i]


@pytest.mark.parametrize("h", [1e-9, 3e-13, 1e-30, 2.0e25])
@pytest.mark.parametrize("dim,degree,stretch,mode", [
    (2, 1, 1.0, 4), (2, 2, 1.7, 5), (3, 1, 1.0, 4), (3, 1, 1.7, 5), (3, 2, 1.0, 4), (3, 2, 0.6, 5),
])
def test_cells_of_any_size(gpu_lib, monkeypatch, dim, degree, stretch, mode, h):
    """A grid in nanometres given in metres, and farther out: the lane kernel is offered and is as exact."""
    monkeypatch.setenv("PPF_CONTRACTION_MODE", str(mode))
    sub = (5, 4, 3)[:dim] + (1,) * (3 - dim)
    wl = W.cahn_hilliard_3d(refine=0, degree=degree, dim=dim, size=1.0, subdivisions=sub, dt=1e-2 * h * h)
    wl.constants = [1.0, 1.5 * h * h, 4.0]
    wl.mesh.size = tuple(n * h * stretch ** d for d, n in enumerate(sub))
    p, o = wl.make_problem(), po.Oracle(wl)
    rng = np.random.default_rng(9)
    c, mu = rng.uniform(0.2, 0.8, p.n_nodes), rng.uniform(-1, 1, p.n_nodes)
    for f, v, age in ((0, c, 0), (0, c, 1), (1, mu, 1)):
        p.upload(f, v, age=age)
        o.set(f, v, age=age)
    for b in (0, 1):
        assert rel_l2(p.apply(b, 0, None, scale=1), o.apply(b, 0, None, scale=1)) < 1e-12, b
        assert p.contraction_mode(b, 0) == mode
    wl = elasticity(dim, degree, tuple(h * stretch ** d for d in range(dim)))
    p, o = wl.make_problem(), po.Oracle(wl)
    u = rng.normal(size=p.field_length(0)) * h
    for scale in (0, 2):
        got, ref = p.apply(0, 1, u, scale=scale), o.apply(0, 1, u, scale=scale)
        assert rel_l2(got, ref, np.abs(ref).max()) < 1e-12
    assert p.contraction_mode(0, 1) == mode
