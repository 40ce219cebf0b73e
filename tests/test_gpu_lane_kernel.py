"""The lane kernel (include/prismspf/gpu/cell_kernel_lanes.cuh) on stretched cells (contraction mode
5) and with several output components, at the smallest meshes, partial tiles and every degree it
covers, against the oracle: one apply within 1e-12 relative L2, steps within 1e-9 (the bars of
tests/test_gpu_fixed_point.py); fields 1e+-150 from O(1) and non-finite values as on cubic cells."""
import os

import numpy as np
import pytest

from oracle import pyoracle as po
from phasefield_gb300 import capi
from phasefield_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def stretched(dim, degree, sub, size, periodic=True):
    wl = W.cahn_hilliard_3d(refine=0, degree=degree, dim=dim, size=1.0, subdivisions=sub, periodic=periodic, dt=1e-6)
    wl.mesh.size = size
    return wl


@pytest.mark.parametrize("dim,degree,sub,size", [
    (2, 1, (1, 1, 1), (1.0, 0.3, 1.0)), (2, 1, (33, 2, 1), (5.0, 4.0, 1.0)),
    (2, 2, (1, 3, 1), (0.7, 9.0, 1.0)), (2, 2, (11, 6, 1), (8.0, 3.0, 1.0)),
    (3, 1, (1, 1, 1), (1.0, 2.0, 0.25)), (3, 1, (5, 7, 3), (5.0, 6.0, 7.0)),
    (3, 2, (1, 2, 1), (3.0, 0.5, 11.0)), (3, 2, (4, 3, 6), (8.0, 5.0, 3.0)),
])
@pytest.mark.parametrize("scale", [1.0, 1e150, 1e-150])
def test_stretched_cells(gpu_lib, monkeypatch, dim, degree, sub, size, scale):
    monkeypatch.setenv("PPF_CONTRACTION_MODE", "5")
    wl = stretched(dim, degree, sub, size, periodic=min(sub[:dim]) > 1)
    p, o = wl.make_problem(), po.Oracle(wl)
    rng = np.random.default_rng(5)
    c, mu = rng.uniform(0.2, 0.8, p.n_nodes), rng.uniform(-1, 1, p.n_nodes) * scale
    for f, v, age in ((0, c, 0), (0, c, 1), (1, mu, 1)):
        p.upload(f, v, age=age)
        o.set(f, v, age=age)
    for b in ((0, 1) if scale == 1.0 else (0,)):
        assert rel_l2(p.apply(b, 0, None, scale=1), o.apply(b, 0, None, scale=1)) < 1e-12, b
        assert p.contraction_mode(b, 0) == 5
    if scale == 1.0:
        p, o = wl.make_problem(), po.Oracle(wl)
        p.solve(4)
        assert o.run(4) == 0
        assert rel_l2(p.download(0, age=1), o.get(0, 1)) < 1e-9


def test_nonfinite_values_on_stretched_cells(gpu_lib, monkeypatch):
    monkeypatch.setenv("PPF_CONTRACTION_MODE", "5")
    wl = stretched(3, 2, (4, 3, 6), (8.0, 5.0, 3.0))
    for bad in (np.nan, np.inf, -np.inf):
        p = wl.make_problem()
        c = wl.initial[0].copy()
        c[c.size // 2] = bad
        p.upload(0, c)
        with pytest.raises(capi.PPFError) as e:
            p.solve(2)
        assert e.value.code == capi.PPF_ERR_NAN
        p.close()


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("size", [(32.0, 32.0, 1.0), (32.0, 21.0, 1.0)])
def test_two_components_and_vectors(gpu_lib, monkeypatch, degree, size):
    """Two scalar fields in a block (and a post-processing block of two), and a vector field."""
    monkeypatch.setenv("PPF_CONTRACTION_MODE", "4" if size[0] == size[1] else "5")
    wl = W.coupled_acch_2d(refine=3, degree=degree, size=32.0, dt=1e-4, n_precip=3)
    wl.mesh.size = size
    p, o = wl.make_problem(), po.Oracle(wl)
    p.solve(6, output_every=6)
    assert o.run(6, 6) == 0
    for f, age in ((0, 1), (1, 1), (2, 0), (3, 0)):
        assert rel_l2(p.download(f, age=age), o.get(f, age)) < 1e-9, f
    assert p.contraction_mode(0, 0) == (4 if size[0] == size[1] else 5)
    wl = W.eshelby_3d(refine=1, degree=degree, size=8.0, n_incl=2)
    wl.mesh.size = (8.0, size[1] / 4, 8.0)
    p, o = wl.make_problem(), po.Oracle(wl)
    u = np.random.default_rng(2).normal(size=p.field_length(0))
    for which, src in ((0, None), (1, u)):
        assert rel_l2(p.apply(0, which, src, scale=0), o.apply(0, which, src, scale=0)) < 1e-12, which
