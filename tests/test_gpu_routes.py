"""The routes that a launch takes by its sizes and components, at the sizes where each can go wrong:
the diagonal probe, the level transfers, the FP32 lane kernel, tiles of small meshes, captured
graphs of several rotation periods, a caller's own capture, ensemble tiles with odd cell counts and
inclusions far from most points. Against the oracle with the bars of the neighbouring tests: one
product or diagonal within 1e-12 relative L2 (sums of at most a few hundred FP64 terms, each
rounded to 1.1e-16), steps within 1e-9, linear solutions within 1e-8 (both sides stop at an absolute
residual of 1e-10 of the scaled system)."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po
from phasefield_gb300 import capi
from phasefield_gb300 import ensemble as E
from phasefield_gb300 import workloads as W
from phasefield_gb300.problem import RectangularMesh

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def elasticity(dim, degree, sub, refine=0, periodic=(0, 0, 0), size=16.0, n_incl=4):
    wl = W.eshelby_3d(refine=0, degree=degree, size=size, n_incl=n_incl, dim=dim)
    wl.mesh = RectangularMesh(dim=dim, degree=degree, size=(size,) * dim + (1.0,) * (3 - dim),
                              subdivisions=sub + (1,) * (3 - len(sub)), global_refinement=refine, periodic=periodic)
    return wl


@pytest.mark.parametrize("dim,degree,sub", [
    (2, 1, (1, 1)), (2, 2, (5, 3)), (2, 3, (3, 4)), (2, 4, (2, 3)),
    (3, 1, (3, 1, 5)), (3, 2, (3, 4, 2)), (3, 3, (2, 1, 3)), (3, 4, (1, 2, 1)),
])
@pytest.mark.parametrize("periodic", [0, 1])
def test_diagonal_probe(gpu_lib, dim, degree, sub, periodic):
    wl = elasticity(dim, degree, sub, periodic=(0, periodic, 0) if sub[1] > 1 else (0, 0, 0))
    p, o = wl.make_problem(), po.Oracle(wl)
    assert rel_l2(p.lhs_diagonal(0), o.diagonal(0)) < 1e-12


@pytest.mark.parametrize("degree", [1, 2, 3])
def test_diagonal_probe_with_other_dependencies(gpu_lib, degree):
    """The Jacobian reads n next to the change (the oracle's probe takes n as zero, so the reference is
    the diagonal of its products)."""
    wl = W.allen_cahn_implicit_2d(refine=3, degree=degree, dt=0.7)
    p, o = wl.make_problem(), po.Oracle(wl)
    p.set_linear_params(0, tolerance_type=0)
    p.upload(0, wl.initial[0])
    o.set(0, wl.initial[0])
    ref = np.array([o.apply(0, 1, e, scale=0)[i] for i, e in enumerate(np.eye(p.n_nodes))])
    assert rel_l2(p.lhs_diagonal(0), ref) < 1e-12


@pytest.mark.parametrize("dim,degree,sub,refine,periodic", [
    (2, 1, (3, 5), 2, (0, 0, 0)), (2, 2, (2, 3), 2, (0, 1, 0)), (2, 3, (1, 2), 2, (0, 0, 0)), (2, 3, (2, 2), 2, (0, 1, 0)),
    (3, 1, (1, 2, 3), 2, (0, 1, 1)), (3, 2, (1, 1, 2), 2, (0, 0, 1)),
])
def test_multigrid_transfers_and_fp32_products(gpu_lib, dim, degree, sub, refine, periodic):
    wl = elasticity(dim, degree, sub, refine, periodic)
    prm = dict(tolerance_type=1, tolerance=1e-10, max_iterations=1500, preconditioner=2, mg_depth=3, smoother_degree=4)
    o = po.Oracle(wl)
    o.set_linear_params(0, **prm)
    rc, oits, _ = o.linear_solve(0)
    for mixed in (0, 1):
        p = wl.make_problem()
        p.set_linear_params(0, mixed_precision=mixed, **prm)
        if rc:  # the V-cycle does not contract on stretched cubic elements: here neither
            assert rc == capi.PPF_ERR_NOCONV and dim == 2 and degree == 3
            with pytest.raises(capi.PPFError) as e:
                p.linear_solve(0)
            assert e.value.code == capi.PPF_ERR_NOCONV
            continue
        its, res = p.linear_solve(0)
        assert res < 1e-10
        assert its <= (1.5 * oits + 2 if mixed else oits + max(2, 0.1 * oits))
        assert rel_l2(p.download(0), o.get(0)) < 1e-8, mixed


@pytest.mark.parametrize("mode", ["1", "2", "3"])
@pytest.mark.parametrize("dim,degree,sub", [(2, 1, (1, 1, 1)), (2, 1, (67, 3, 1)), (2, 2, (3, 5, 1)), (2, 3, (5, 2, 1)),
                                            (3, 1, (3, 2, 5)), (3, 2, (2, 3, 1)), (3, 4, (1, 2, 1))])
def test_tiles_of_small_meshes(gpu_lib, monkeypatch, mode, dim, degree, sub):
    monkeypatch.setenv("PPF_CONTRACTION_MODE", mode)
    wl = W.cahn_hilliard_3d(refine=0, degree=degree, dim=dim, size=4.0, subdivisions=sub, periodic=min(sub[:dim]) > 1,
                            dt=1e-6)
    wl.mesh.size = tuple(float(s) for s in sub)
    p, o = wl.make_problem(), po.Oracle(wl)
    p.solve(4)
    assert o.run(4) == 0
    for f in (0, 1):
        assert rel_l2(p.download(f, age=1 - f), o.get(f, 1 - f)) < 1e-9, f


@pytest.mark.parametrize("runs", [(1,), (2, 3), (16, 1), (7, 9, 11), (40,)])
def test_graphs_of_several_periods(gpu_lib, runs):
    """Runs shorter and longer than a captured graph, resumed at every phase of the rotation."""
    wl = W.coupled_acch_2d(refine=3, degree=1, size=32.0, dt=1e-3, n_precip=3)
    res = []
    for use_graph in (0, 1):
        p = wl.make_problem()
        p.lib.ppf_set_use_graph(p.h, use_graph)
        for n in runs:
            p.solve(n)
        res.append([p.download(f, age=1) for f in (0, 1)] + [np.array(p.get_time())])
        p.close()
    for a, b in zip(*res):
        assert rel_l2(b, a) < 1e-12


def test_product_in_a_caller_capture(gpu_lib):
    """A captured ppf_apply_device may be replayed any number of times, between plain calls."""
    import torch

    wl = elasticity(3, 2, (3, 4, 2))
    p, o = wl.make_problem(), po.Oracle(wl)
    u = np.random.default_rng(3).normal(size=p.field_length(0))
    ref = o.apply(0, 1, u, scale=0)
    src = torch.from_numpy(u).cuda()
    dst = torch.zeros_like(src)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    p._check(p.lib.ppf_set_stream(p.h, C.c_void_p(s.cuda_stream)))
    call = lambda: p._check(p.lib.ppf_apply_device(p.h, 0, 1, src.data_ptr(), dst.data_ptr(), 0))
    for warm in (1, 2):  # an odd and an even number of products before the capture
        with torch.cuda.stream(s):
            for _ in range(warm):
                call()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            call()
        for _ in range(3):
            with torch.cuda.stream(s):
                dst.fill_(float("nan"))
                g.replay()
                s.synchronize()
                assert rel_l2(dst.cpu().numpy(), ref) < 1e-12
                dst.fill_(float("nan"))
                call()
                s.synchronize()
                assert rel_l2(dst.cpu().numpy(), ref) < 1e-12
    p._check(p.lib.ppf_set_stream(p.h, None))


@pytest.mark.parametrize("tune", [False, True])
@pytest.mark.parametrize("copies", [1, 20, 160])
@pytest.mark.parametrize("degree", [1, 2])
def test_ensemble_tiles(gpu_lib, degree, copies, tune):
    """Instances of one cell, of one row, and just past a warp's width or a tile's height, as few as
    run on one thread per point and as many as take either lane layout."""
    subs = [(1, 1), (31, 1), (1, 33), (32, 5), (33, 7), (29, 13), (3, 19)]
    h = 2.0
    meshes = [RectangularMesh(dim=2, degree=degree, size=(h * a, h * b, 1.0), subdivisions=(a, b, 1)) for a, b in subs]
    rng = np.random.default_rng(degree)
    ics = [rng.uniform(0.0, 1.0, size=int(np.prod(m.nodes))) for m in meshes]
    dt, steps = 0.01, 5
    # (a spare Q1 or Q2 instance, so that a launch holds both degrees)
    other = RectangularMesh(dim=2, degree=3 - degree, size=(h * 9, h * 4, 1.0), subdivisions=(9, 4, 1))
    ens = E.Ensemble(meshes * copies + [other], [1.0] * (len(subs) * copies + 1), [2.0] * (len(subs) * copies + 1), dt)
    for i in range(len(subs) * copies):
        ens.upload(i, ics[i % len(subs)])
    ens.upload(len(subs) * copies, np.zeros(int(np.prod(other.nodes))))
    if tune:
        ens.autotune(steps=1)  # runs every tile shape and grid
    ens.run(steps, use_graph=True)
    for i, m in enumerate(meshes):
        wl = W.allen_cahn_2d(refine=0, degree=degree, m_well=1.0, kappa=2.0, dt=dt, subdivisions=subs[i])
        wl.mesh, wl.initial = m, {0: ics[i]}
        o = po.Oracle(wl)
        assert o.run(steps) == 0
        for j in (i, len(subs) * (copies - 1) + i):
            assert rel_l2(ens.download(j), o.get(0, 1)) < 1e-9, (subs[i], j)
    assert np.all(ens.download(len(subs) * copies) == 0.0)


@pytest.mark.parametrize("runs", [(2,), (30, 5, 24), (7, 7, 7)])
def test_ensemble_graphs(gpu_lib, runs):
    """Runs from every phase of the accumulator rotation, shorter and longer than a captured graph."""
    meshes, mw, ka, ics = E.allen_cahn_ensemble(n_instances=5, min_cells=8, max_cells=24, seed=3)
    res = []
    for use_graph in (False, True):
        ens = E.Ensemble(meshes, mw, ka, 0.01)
        for i, ic in enumerate(ics):
            ens.upload(i, ic)
        for n in runs:
            ens.run(n, use_graph=use_graph)
        res.append([ens.download(i) for i in range(len(meshes))])
    for a, b in zip(*res):
        assert rel_l2(b, a) < 1e-12


def test_inclusions_ruled_out_by_distance(gpu_lib):
    wl = elasticity(3, 2, (9, 9, 9), size=90.0, n_incl=40)  # most of the 40 are out of reach of a point
    p, o = wl.make_problem(), po.Oracle(wl)
    assert rel_l2(p.apply(0, 0, None, scale=0), o.apply(0, 0, None, scale=0)) < 1e-12
