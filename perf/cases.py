"""The work a user of the engine has it do, as measurable cases.

A case is a plain dict; ``kind`` names the path and the other entries its sizes and options:

  step       one allocation-free Allen-Cahn step on the caller's device vectors
  explicit   increments of an explicit simulation between two outputs (Allen-Cahn in 2-D,
             Cahn-Hilliard in 2-D and 3-D, cubic and stretched cells, periodic and natural faces)
  apply      one evaluation of the elasticity operator (a matrix-free product, scaled or not)
  gmg        two load steps of a linear elasticity problem by GMG-preconditioned CG, in FP64 or
             with the FP32 smoothing levels
  newton     implicit Allen-Cahn increments (Newton with Chebyshev-preconditioned CG inside)
  ensemble   steps of a batch of independent simulations, then their fields
  amr        increments on an adaptive mesh between two remeshings
  adjoint    a checkpointed forward sweep and the gradient of a loss back through it

``listed`` has the sizes of the benchmark, of its configurations and some odd ones; ``draw``
gives others of the same ranges. Inputs come from the seed alone and are made on the GPU.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from phasefield_gb300 import capi
from phasefield_gb300 import workloads as W
from phasefield_gb300.ensemble import Ensemble
from phasefield_gb300.problem import FieldAttributes, Problem, RectangularMesh, Vector

DEV = "cuda"


def listed():
    return [
        # the smallest call: one step of a small 2-D mesh, launches and host work only
        dict(name="step_2d_q1_64", kind="step", dim=2, degree=1, nx=64, ny=64, nz=1, size=100.0),
        # the Allen-Cahn benchmark configuration (128^2 Q1), 100 increments between outputs
        dict(name="allen_cahn_2d_q1_128", kind="explicit", model="allen_cahn", dim=2, degree=1, nx=128, ny=128, nz=1,
             h=0.78125, stretch=0.0, periodic=False, increments=100),
        # the headline: Cahn-Hilliard 64^3 Q2, periodic
        dict(name="cahn_hilliard_3d_q2_64", kind="explicit", model="cahn_hilliard", dim=3, degree=2, nx=64, ny=64,
             nz=64, h=1.0, stretch=0.0, periodic=True, increments=10),
        # an odd box with natural faces and cells that are not cubes
        dict(name="cahn_hilliard_3d_q2_odd", kind="explicit", model="cahn_hilliard", dim=3, degree=2, nx=37, ny=52,
             nz=29, h=1.0, stretch=0.08, periodic=False, increments=10),
        # the largest: 17 million nodes a field
        dict(name="cahn_hilliard_3d_q2_128", kind="explicit", model="cahn_hilliard", dim=3, degree=2, nx=128, ny=128,
             nz=128, h=1.25, stretch=0.0, periodic=True, increments=10),
        # a matrix-free product of the vector-valued elasticity operator, as a caller's own solver asks for it
        dict(name="elasticity_apply_q2_48", kind="apply", dim=3, degree=2, nx=48, ny=48, nz=48, h=1.0, scale=2),
        # the elasticity benchmark configuration at half its edge, all levels in FP64
        dict(name="gmg_fp64_q2_32", kind="gmg", degree=2, sub=1, refine=5, mixed=0),
        # the elasticity benchmark configuration (64^3 Q2, 6.4 million unknowns), FP32 smoothing levels
        dict(name="gmg_mixed_q2_64", kind="gmg", degree=2, sub=1, refine=6, mixed=1),
        # implicit time stepping at a step far above the explicit limit
        dict(name="newton_2d_q2_64", kind="newton", degree=2, nx=64, ny=64, increments=3),
        # a calibration batch: uneven meshes, both degrees
        dict(name="ensemble_48", kind="ensemble", count=48, min_cells=32, max_cells=256, steps=150),
        # the adaptive Allen-Cahn application (levels 3 to 8, Q1) between two remeshings
        dict(name="amr_2d_q1", kind="amr", degree=1, refine=8, min_level=3, increments=100),
        # gradient of a loss through 40 steps with 8 snapshots
        dict(name="adjoint_2d_q2_128", kind="adjoint", degree=2, nx=128, ny=128, steps=40, snapshots=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "explicit", "explicit", "explicit", "apply", "gmg", "newton", "ensemble", "amr",
                       "adjoint"])
    degree = rng.choice([1, 2, 2])
    if kind == "step":
        dim = rng.choice([2, 2, 3])
        n = [_log_int(rng, 16, 200) if dim == 2 else _log_int(rng, 6, 40) for _ in range(3)]
        return dict(kind=kind, dim=dim, degree=degree, nx=n[0], ny=n[1], nz=n[2] if dim == 3 else 1,
                    size=round(rng.uniform(20.0, 120.0), 2))
    if kind == "explicit":
        model = rng.choice(["allen_cahn", "cahn_hilliard", "cahn_hilliard"])
        dim = 2 if model == "allen_cahn" else rng.choice([2, 3, 3])
        n = [_log_int(rng, 24, 400) if dim == 2 else _log_int(rng, 12, 96) for _ in range(3)]
        return dict(kind=kind, model=model, dim=dim, degree=degree, nx=n[0], ny=n[1], nz=n[2] if dim == 3 else 1,
                    h=rng.choice([1.0, round(rng.uniform(0.95, 1.6), 4)]), stretch=rng.choice([0.0, 0.05, 0.1]),
                    periodic=rng.random() < 0.5, increments=100 if dim == 2 else 10)
    if kind == "apply":
        n = [_log_int(rng, 8, 64) for _ in range(3)]
        return dict(kind=kind, dim=3, degree=degree, nx=n[0], ny=n[1], nz=n[2], h=round(rng.uniform(0.5, 2.0), 3),
                    scale=rng.choice([0, 2]))
    if kind == "gmg":
        sub, refine = rng.choice([(1, 4), (1, 5), (3, 3), (3, 4), (5, 3), (2, 5), (7, 3)])
        return dict(kind=kind, degree=degree, sub=sub, refine=refine, mixed=rng.choice([0, 1]))
    if kind == "newton":
        return dict(kind=kind, degree=degree, nx=_log_int(rng, 20, 128), ny=_log_int(rng, 20, 128), increments=3)
    if kind == "ensemble":
        lo = _log_int(rng, 16, 64)
        return dict(kind=kind, count=rng.randint(8, 48), min_cells=lo, max_cells=lo * rng.randint(2, 4),
                    steps=rng.randint(60, 150))
    if kind == "amr":
        return dict(kind=kind, degree=degree, refine=rng.randint(6, 8), min_level=3, increments=2 * rng.randint(25, 60))
    return dict(kind="adjoint", degree=degree, nx=_log_int(rng, 32, 160), ny=_log_int(rng, 32, 160),
                steps=rng.randint(20, 40), snapshots=rng.randint(4, 8))


# ---------------------------------------------------------------------------------------------
# descriptions
# ---------------------------------------------------------------------------------------------
class State:
    pass


def _cells(case):
    return tuple(int(case[k]) for k in ("nx", "ny", "nz")[:case.get("dim", 2)])


def _sizes(case):
    """Edge lengths of the box: cubes of edge h, or stretched along the later axes."""
    cells, s = _cells(case), case.get("stretch", 0.0)
    return tuple(n * case["h"] * (1.0 + s * d) for d, n in enumerate(cells))


def _mesh(cells, sizes, degree, periodic=False):
    dim = len(cells)
    fill = 3 - dim
    return RectangularMesh(dim=dim, degree=degree, size=tuple(sizes) + (1.0,) * fill,
                           subdivisions=tuple(cells) + (1,) * fill, global_refinement=0,
                           periodic=(int(periodic),) * dim + (0,) * fill)


def _axis(cells, size, degree):
    """Node coordinates along one axis."""
    gl = np.array([0.0, 1.0]) if degree == 1 else np.array([0.0, 0.5, 1.0])
    i = np.arange(degree * cells + 1)
    c = np.minimum(i // degree, cells - 1)
    return torch.tensor((c + gl[i - degree * c]) * (size / cells), dtype=torch.float64, device=DEV)


def _grains(cells, sizes, degree, rng, count=12, lo=5.0, hi=15.0, width=2.0):
    """Seeded grains: min(1, sum of tanh profiles), on the lattice (slowest axis first)."""
    axes = [_axis(c, s, degree) for c, s in zip(cells, sizes)]
    grid = torch.meshgrid(*reversed(axes), indexing="ij")[::-1]
    scale = min(sizes) / 100.0
    out = torch.zeros_like(grid[0])
    for _ in range(count):
        r2 = 0.0
        for d, g in enumerate(grid):
            r2 = r2 + (g - rng.uniform(0.0, sizes[d])) ** 2
        out += 0.5 * (1.0 - torch.tanh((torch.sqrt(r2) - rng.uniform(lo, hi) * scale) / (width * scale)))
    return torch.clamp(out, max=1.0)


def _smooth_noise(shape, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return 0.5 + 0.05 * (2.0 * torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) - 1.0)


def _lattice_shape(cells, degree):
    return tuple(degree * c + 1 for c in reversed(cells))


def _explicit(case, seed):
    """Mesh, initial field, time step and constants of an explicit case."""
    cells, sizes, k = _cells(case), _sizes(case), case["degree"]
    hmin = min(s / n for s, n in zip(sizes, cells))
    rng = np.random.default_rng(seed)
    if case["model"] == "allen_cahn":
        return cells, sizes, _grains(cells, sizes, k, rng), min(0.01, 0.01 * hmin * hmin), [1.0, 2.0]
    return cells, sizes, _smooth_noise(_lattice_shape(cells, k), seed), 1e-4 * min(1.0, hmin ** 4), [1.0, 1.5, 4.0]


def _own_stream(problem):
    """Queues a problem's work on a stream that torch knows, so that device copies are in order."""
    s = torch.cuda.Stream()
    problem._check(problem.lib.ppf_set_stream(problem.h, C.c_void_p(s.cuda_stream)))
    return s


def _keep(problem, ages):
    """Copies of the state vectors of the given (field, age) pairs."""
    return {fa: problem.device_view(*fa).clone() for fa in ages}


def _restore(state):
    """The state as it was kept: what a program does that goes on from a checkpoint."""
    with torch.cuda.stream(state.stream):
        for fa, v in state.kept.items():
            state.problem.device_view(*fa).copy_(v)
    state.problem.set_time(*state.time)


def _results(state, ages):
    """The solved fields, copied out of the state the next increments overwrite."""
    with torch.cuda.stream(state.stream):
        return [state.problem.device_view(*fa).clone() for fa in ages]


def _stiffness():
    """Voigt stiffness of a cubic crystal."""
    C6 = np.zeros((6, 6))
    C6[:3, :3] = 150.0
    np.fill_diagonal(C6, [250.0] * 3 + [100.0] * 3)
    return C6


_EIGENSTRAIN, _WIDTH = 0.01, 1.0


def _inclusions(size, seed):
    """Centres and radii (x, y, z, r) of spherical inclusions with an eigenstrain."""
    rng = np.random.default_rng(seed)
    count = 40 if size >= 48 else 8
    return np.concatenate([rng.uniform(0.0, size, (count, 3)), rng.uniform(0.05 * size, 0.1 * size, (count, 1))], 1)


def _elasticity_problem(cells, h, degree, seed, dirichlet, sub=None, refine=0):
    incl = _inclusions(cells[0] * h, seed)
    constants = [*_stiffness().ravel(), _EIGENSTRAIN, _WIDTH, float(len(incl)), *incl.ravel()]
    mesh = RectangularMesh(dim=3, degree=degree, size=tuple(c * h for c in cells), subdivisions=tuple(sub or cells),
                           global_refinement=refine)
    fields = [FieldAttributes("u", Vector, dirichlet=dirichlet)]
    return Problem(fields, W.eshelby_3d(refine=0, degree=degree).blocks, mesh, "eshelby", constants, 0.0)


def _gmg_cells(case):
    return (case["sub"] << case["refine"],) * 3


def _acch(case, seed):
    cells, k = _cells(case), case["degree"]
    rng = np.random.default_rng(seed)
    sizes = tuple(0.5 * c for c in cells)
    n0 = _grains(cells, sizes, k, rng, count=8, lo=6.0, hi=14.0, width=1.5)
    return cells, sizes, 0.009 + (0.125 - 0.009) * n0, n0, 2e-4, [1.0, 1.0, 2.0]


def _ensemble(case, seed):
    # the batch's meshes are the case's, its parameters and initial fields the seed's
    sizes, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed)
    meshes, mw, ka, ics = [], [], [], []
    for _ in range(case["count"]):
        n = int(sizes.integers(case["min_cells"], case["max_cells"] + 1))
        degree = int(sizes.integers(1, 3))
        meshes.append(_mesh((n, n), (100.0, 100.0), degree))
        mw.append(float(rng.uniform(0.5, 2.0)))
        ka.append(float(rng.uniform(1.0, 4.0)))
        ics.append(_grains((n, n), (100.0, 100.0), degree, rng))
    hmin = min(100.0 / m.subdivisions[0] for m in meshes)
    return meshes, np.array(mw), np.array(ka), ics, min(0.01, 0.004 * hmin * hmin)


# ---------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return state.run(state)


def _prepare_step(case, seed):
    s = State()
    s.run = _run_step
    s.lib = capi.load()
    cells = _cells(case)
    sizes = tuple(case["size"] * n / cells[0] for n in cells)
    m = capi.MeshDesc()
    m.dim, m.degree, m.global_refinement = len(cells), case["degree"], 0
    for d in range(3):
        m.subdivisions[d] = cells[d] if d < len(cells) else 1
        m.size[d] = sizes[d] if d < len(cells) else 1.0
    s.mesh = m
    s.n_old = _grains(cells, sizes, case["degree"], np.random.default_rng(seed)).reshape(-1)
    s.n_new = torch.empty_like(s.n_old)
    s.stream = torch.cuda.current_stream().cuda_stream
    return s


def _run_step(s):
    rc = s.lib.ppf_allen_cahn_step_noalloc(C.byref(s.mesh), 1.0, 2.0, 0.001, s.n_old.data_ptr(), s.n_new.data_ptr(),
                                           s.stream)
    if rc:
        raise RuntimeError("step failed: %d" % rc)
    return s.n_new


def _prepare_explicit(case, seed):
    s = State()
    s.run = _run_explicit
    cells, sizes, u0, dt, consts = _explicit(case, seed)
    k, periodic = case["degree"], case["periodic"]
    if case["model"] == "allen_cahn":
        wl = W.allen_cahn_2d(refine=0, degree=k)
        s.solved = [(0, 1)]
    else:
        wl = W.cahn_hilliard_3d(refine=0, degree=k, dim=len(cells))
        s.solved = [(0, 1), (1, 1)]
    p = Problem(wl.fields, wl.blocks, _mesh(cells, sizes, k, periodic), wl.model, consts, dt)
    s.problem, s.stream = p, _own_stream(p)
    p.upload(0, u0.reshape(-1).cpu().numpy())
    p.solve(1)  # the initial condition and the first increment
    s.kept, s.time = _keep(p, s.solved), p.get_time()
    s.until = 1 + case["increments"]
    return s


def _run_explicit(s):
    _restore(s)
    s.problem.solve(s.until)
    return _results(s, s.solved)


def _prepare_apply(case, seed):
    s = State()
    s.run = _run_apply
    cells = _cells(case)
    p = _elasticity_problem(cells, case["h"], case["degree"], seed, {(c, 0): 0.0 for c in range(3)})
    s.problem, s.stream, s.scale = p, _own_stream(p), case["scale"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    s.src = torch.randn(p.field_length(0), generator=g, device=DEV, dtype=torch.float64)
    s.dst = torch.empty_like(s.src)
    torch.cuda.synchronize()
    p._check(p.lib.ppf_apply_device(p.h, 0, 1, s.src.data_ptr(), s.dst.data_ptr(), s.scale))
    return s


def _run_apply(s):
    p = s.problem
    p._check(p.lib.ppf_apply_device(p.h, 0, 1, s.src.data_ptr(), s.dst.data_ptr(), s.scale))
    return s.dst


# the box is held at x = 0 and its far face moved along x: two displacements a pass
_GMG_H = 1.0
_GMG_LOADS = (0.05, -0.03)


def _prepare_gmg(case, seed):
    s = State()
    s.run = _run_gmg
    cells = _gmg_cells(case)
    dirichlet = {(c, 0): 0.0 for c in range(3)}
    dirichlet[(0, 1)] = _GMG_LOADS[0]
    p = _elasticity_problem(cells, _GMG_H, case["degree"], seed, dirichlet, (case["sub"],) * 3, case["refine"])
    s.problem, s.stream = p, _own_stream(p)
    norm = float(np.linalg.norm(p.apply(0, 0, None, scale=0)))
    p.set_linear_params(0, tolerance_type=0, tolerance=1e-12 * norm, max_iterations=500, preconditioner=2,
                        mg_depth=case["refine"] + 1, smoother_degree=4, mixed_precision=case["mixed"])
    shape = (3,) + _lattice_shape(cells, case["degree"])
    s.loads = []
    for g in _GMG_LOADS:
        v = np.zeros(shape)
        v[0, :, :, -1] = g
        s.loads.append(v.reshape(-1))
    return s


def _run_gmg(s):
    p, out = s.problem, []
    for load in s.loads:
        p._check(p.lib.ppf_set_dirichlet_values(p.h, 0, capi.dptr(load)))
        p.linear_solve(0)
        out += _results(s, [(0, 0)])
    return out


def _prepare_newton(case, seed):
    s = State()
    s.run = _run_explicit
    cells, k = _cells(case), case["degree"]
    sizes = tuple(100.0 * c / max(cells) for c in cells)
    wl = W.allen_cahn_implicit_2d(refine=0, degree=k)
    p = Problem(wl.fields, wl.blocks, _mesh(cells, sizes, k), wl.model, [1.0, 2.0], 0.5)
    p.set_linear_params(0, tolerance_type=1, tolerance=1e-12, max_iterations=3000, preconditioner=1, smoother_degree=4)
    p.set_newton_params(0, max_iterations=50, tolerance=1e-11)
    s.problem, s.stream = p, _own_stream(p)
    p.upload(0, _grains(cells, sizes, k, np.random.default_rng(seed)).reshape(-1).cpu().numpy())
    p.solve(1)
    s.solved = [(0, 1)]
    s.kept, s.time = _keep(p, s.solved), p.get_time()
    s.until = 1 + case["increments"]
    return s


def _prepare_ensemble(case, seed):
    s = State()
    s.run = _run_ensemble
    meshes, mw, ka, ics, dt = _ensemble(case, seed)
    s.ensemble, s.steps = Ensemble(meshes, mw, ka, dt), case["steps"]
    for i, v in enumerate(ics):
        s.ensemble.upload(i, v.reshape(-1).cpu().numpy())
    return s


def _run_ensemble(s):
    # a pass goes on from the fields of the last one
    s.ensemble.run(s.steps)
    return [s.ensemble.download(i) for i in range(len(s.ensemble.meshes))]


def _prepare_amr(case, seed):
    s = State()
    s.run = _run_explicit
    wl = W.allen_cahn_amr_2d(refine=case["refine"], degree=case["degree"], min_level=case["min_level"],
                             max_level=case["refine"], period=800, n_grains=12,
                             dt=min(0.01, 0.01 * (100.0 / 2 ** case["refine"]) ** 2))
    p = wl.make_problem()
    s.problem, s.stream = p, _own_stream(p)
    p.solve(1)
    s.solved = [(0, 1)]
    s.kept, s.time = _keep(p, s.solved), p.get_time()
    # the mesh is the case's; the order parameter of its grains, that of the seed
    with torch.cuda.stream(s.stream):
        s.kept[(0, 1)] *= np.random.default_rng(seed).uniform(0.9, 1.0)
    s.until = 1 + case["increments"]
    return s


def _prepare_adjoint(case, seed):
    s = State()
    s.run = _run_adjoint
    cells, sizes, c0, n0, dt, consts = _acch(case, seed)
    wl = W.coupled_acch_2d(refine=0, degree=case["degree"])
    p = Problem(wl.fields, wl.blocks, _mesh(cells, sizes, case["degree"]), wl.model, consts, dt)
    s.problem, s.stream = p, _own_stream(p)
    s.start = [c0.reshape(-1).contiguous(), n0.reshape(-1).contiguous()]
    s.weights = _adjoint_weights(c0.numel(), seed)
    s.steps, s.snapshots = case["steps"], case["snapshots"]
    torch.cuda.synchronize()
    return s


def _adjoint_weights(n, seed):
    """dJ/du at the last step: the residual of a fit, of both signs."""
    return np.random.default_rng(seed + 1).normal(size=2 * n)


def _run_adjoint(s):
    p = s.problem
    with torch.cuda.stream(s.stream):
        for f, v in enumerate(s.start):
            p.device_view(f).copy_(v)
    p.adjoint_forward(0, s.steps, s.snapshots)
    c, n = _results(s, [(0, 0), (1, 0)])
    params, du0, _ = p.adjoint_backward(s.weights)
    return {"params": params, "du0": du0, "c": c, "n": n}


# ---------------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------------
def _nodes(cells, k):
    return math.prod(k * c + 1 for c in cells)


def _cell_flops(dim, k, rows_in, rows_out, point):
    """Sum-factorised gradients of rows_in rows, integration of rows_out rows, `point` flops a point."""
    n = k + 1
    return n ** dim * (2 * dim * n * (rows_in + rows_out) + point)


def work(case):
    kind, k = case["kind"], case.get("degree", 1)
    if kind in ("step", "newton", "adjoint", "explicit", "apply"):
        cells = _cells(case)
        dim, N, nc = len(cells), _nodes(cells, k), math.prod(cells)
    if kind == "step":
        return {"bytes": 16 * N, "flops": nc * _cell_flops(dim, k, 1, 1, 12)}
    if kind == "explicit":
        if case["model"] == "allen_cahn":
            return {"bytes": 16 * N * case["increments"], "flops": case["increments"] * nc * _cell_flops(dim, k, 1, 1, 12)}
        return {"bytes": 40 * N * case["increments"],
                "flops": case["increments"] * nc * (_cell_flops(dim, k, 1, 1, 8) + _cell_flops(dim, k, 1, 1, 12))}
    if kind == "apply":
        return {"bytes": 48 * N, "flops": nc * _cell_flops(3, k, 3, 3, 45)}
    if kind == "gmg":
        # two solves of about 22 iterations, each an FP64 product and a V-cycle of about 9 products a level
        cells = _gmg_cells(case)
        N, nc, product = _nodes(cells, k), math.prod(cells), _cell_flops(3, k, 3, 3, 45)
        low = 24 if case["mixed"] else 48
        return {"bytes": 2 * 22 * N * (48 + 9 * low * 8 // 7), "flops": 2 * 22 * nc * product * (1 + 9 * 8 / 7)}
    if kind == "newton":
        # about 4 Newton steps of 10 CG iterations with 5 products each, an increment
        return {"bytes": 16 * N * 200 * case["increments"],
                "flops": 200 * case["increments"] * nc * _cell_flops(2, k, 1, 1, 12)}
    if kind == "ensemble":
        mid = 0.5 * (case["min_cells"] + case["max_cells"])
        per = 0.5 * (mid + 1) ** 2 + 0.5 * (2 * mid + 1) ** 2
        flops = 0.5 * mid * mid * (_cell_flops(2, 1, 1, 1, 12) + _cell_flops(2, 2, 1, 1, 12))
        return {"bytes": int(16 * per * case["count"] * case["steps"]), "flops": flops * case["count"] * case["steps"]}
    if kind == "amr":
        # the interfaces hold about an eighth of the finest mesh's cells
        nc = max(64, 4 ** case["refine"] // 8)
        return {"bytes": 16 * nc * k * k * case["increments"],
                "flops": case["increments"] * nc * _cell_flops(2, k, 1, 1, 12)}
    steps = 3 * case["steps"]  # forward, recomputation, reverse
    return {"bytes": 32 * N * steps, "flops": steps * nc * _cell_flops(2, k, 2, 2, 60)}


# ---------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
class _Lattice:
    """Q1/Q2 elements with Gauss-Lobatto collocation on a box, fields as (.., z, y, x) tensors."""

    def __init__(self, cells, sizes, degree, periodic=False):
        self.cells, self.k, self.n, self.dim, self.periodic = cells, degree, degree + 1, len(cells), periodic
        if degree == 1:
            w, D = [0.5, 0.5], [[-1.0, 1.0], [-1.0, 1.0]]
        else:
            w, D = [1 / 6, 4 / 6, 1 / 6], [[-3.0, 4.0, -1.0], [-1.0, 0.0, 1.0], [1.0, -4.0, 3.0]]
        D = torch.tensor(D, dtype=torch.float64, device=DEV)
        w = torch.tensor(w, dtype=torch.float64, device=DEV)
        self.D = [D * (c / s) for c, s in zip(cells, sizes)]
        self.jxw = torch.ones((), dtype=torch.float64, device=DEV)
        for d in range(self.dim):
            wd = (w * (sizes[d] / cells[d])).repeat(cells[d])
            self.jxw = self.jxw * wd.reshape((-1,) + (1,) * d)
        self.mass = self.scatter(self.jxw)

    def split(self, u):
        """Nodal values of every cell: each axis of length k*cells+1 becomes cells*(k+1)."""
        for d in range(self.dim):
            ax = u.dim() - 1 - d
            i = torch.arange(self.cells[d], device=DEV)[:, None] * self.k + torch.arange(self.n, device=DEV)[None, :]
            u = u.index_select(ax, i.reshape(-1))
        return u

    def _line(self, v, d, M):
        ax = v.dim() - 1 - d
        s = list(v.shape)
        x = v.reshape(s[:ax] + [self.cells[d], self.n] + s[ax + 1:]).movedim(ax + 1, -1)
        return torch.matmul(x, M.t()).movedim(-1, ax + 1).reshape(s)

    def grad(self, v):
        return [self._line(v, d, self.D[d]) for d in range(self.dim)]

    def scatter(self, v):
        for d in range(self.dim):
            ax = v.dim() - 1 - d
            s = list(v.shape)
            x = v.reshape(s[:ax] + [self.cells[d], self.n] + s[ax + 1:])
            ends = x.select(ax + 1, self.n - 1)
            pad = torch.zeros_like(ends.narrow(ax, 0, 1))
            first = torch.cat([x.select(ax + 1, 0), pad], ax) + torch.cat([pad, ends], ax)
            if self.periodic:
                first = first.clone()
                both = first.narrow(ax, 0, 1) + first.narrow(ax, self.cells[d], 1)
                first = torch.cat([both, first.narrow(ax, 1, self.cells[d] - 1), both], ax)
            if self.k == 1:
                v = first
            else:
                mid = torch.cat([x.select(ax + 1, 1), pad], ax)
                v = torch.stack([first, mid], ax + 1).reshape(s[:ax] + [2 * (self.cells[d] + 1)] + s[ax + 1:])
                v = v.narrow(ax, 0, 2 * self.cells[d] + 1)
        return v

    def integrate(self, value, grads):
        r = value * self.jxw if value is not None else 0.0
        for d, g in enumerate(grads or []):
            r = r + self._line(g * self.jxw, d, self.D[d].t())
        return self.scatter(r)


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, int(seed)) if f else None


def _exact_step(case, seed):
    cells = _cells(case)
    sizes = tuple(case["size"] * n / cells[0] for n in cells)
    L = _Lattice(cells, sizes, case["degree"])
    u = _grains(cells, sizes, case["degree"], np.random.default_rng(seed))
    return _allen_cahn_step(L, u, 0.001, 1.0, 2.0).reshape(-1)


def _allen_cahn_step(L, u, dt, m, kappa):
    v = L.split(u)
    value = v - dt * m * (4.0 * v * (v - 1.0) * (v - 0.5))
    return L.integrate(value, [-dt * kappa * m * g for g in L.grad(v)]) / L.mass


def _exact_explicit(case, seed):
    cells, sizes, u, dt, consts = _explicit(case, seed)
    if case["increments"] * _nodes(cells, case["degree"]) > 4e8:
        return None
    L = _Lattice(cells, sizes, case["degree"], case["periodic"])
    if case["model"] == "allen_cahn":
        for _ in range(1 + case["increments"]):
            u = _allen_cahn_step(L, u, dt, *consts)
        return [u.reshape(-1)]
    M, K, Wc = consts

    def potential(c):
        v = L.split(c)
        return L.integrate(Wc * v * (v - 1.0) * (v - 0.5), [K * g for g in L.grad(v)]) / L.mass

    mu = potential(u)
    for _ in range(1 + case["increments"]):
        u = L.integrate(L.split(u), [-M * dt * g for g in L.grad(L.split(mu))]) / L.mass
        mu = potential(u)
    return [u.reshape(-1), mu.reshape(-1)]


def _stress(C6, g):
    """Voigt stress of the displacement gradients g[i][j] = du_i/dx_j."""
    e = [g[0][0], g[1][1], g[2][2], g[1][2] + g[2][1], g[0][2] + g[2][0], g[0][1] + g[1][0]]
    s = [sum(float(C6[i, j]) * e[j] for j in range(6) if C6[i, j]) for i in range(6)]
    return [[s[0], s[5], s[4]], [s[5], s[1], s[3]], [s[4], s[3], s[2]]]


def _elasticity(L, C6, u):
    s = _stress(C6, [L.grad(L.split(u[c])) for c in range(3)])
    return torch.stack([L.integrate(None, s[c]) for c in range(3)])


def _exact_apply(case, seed):
    cells = _cells(case)
    L = _Lattice(cells, tuple(c * case["h"] for c in cells), case["degree"])
    shape = (3,) + _lattice_shape(cells, case["degree"])
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    u = torch.randn(math.prod(shape), generator=g, device=DEV, dtype=torch.float64).reshape(shape)
    u[..., 0] = 0.0
    r = _elasticity(L, _stiffness(), u)
    if case["scale"] == 2:
        r = r * torch.sqrt(1.0 / L.mass)
    r[..., 0] = 0.0
    return r.reshape(-1)


def _exact_gmg(case, seed):
    cells, k = _gmg_cells(case), case["degree"]
    if 3 * _nodes(cells, k) > 1_000_000:
        return None
    size = cells[0] * _GMG_H
    L = _Lattice(cells, (size,) * 3, k)
    C6 = _stiffness()
    x = _axis(cells[0], size, k)
    grid = torch.meshgrid(x, x, x, indexing="ij")[::-1]
    strain = torch.zeros_like(grid[0])
    for cx, cy, cz, r in _inclusions(size, seed):
        d = torch.sqrt((grid[0] - cx) ** 2 + (grid[1] - cy) ** 2 + (grid[2] - cz) ** 2)
        strain += 0.5 * (1.0 - torch.tanh((d - r) / _WIDTH))
    e = L.split(_EIGENSTRAIN * torch.clamp(strain, max=1.0))
    zero = torch.zeros_like(e)
    s = _stress(C6, [[e if i == j else zero for j in range(3)] for i in range(3)])
    rhs = torch.stack([L.integrate(None, [-s[c][d] for d in range(3)]) for c in range(3)])
    held = torch.zeros((3,) + tuple(strain.shape), dtype=torch.bool, device=DEV)
    held[..., 0] = True
    held[0, ..., -1] = True

    def free(v):
        return torch.where(held, torch.zeros_like(v), v)

    # CG scaled by the lumped mass
    scale = 1.0 / L.mass
    out = []
    for load in _GMG_LOADS:
        g = torch.zeros_like(rhs)
        g[0, ..., -1] = load
        r = free(rhs - _elasticity(L, C6, g))
        x, z = torch.zeros_like(r), scale * r
        p, rz, stop = z.clone(), (r * z).sum(), 1e-26 * (r * r).sum()
        for _ in range(4000):
            q = free(_elasticity(L, C6, p))
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if (r * r).sum() < stop:
                break
            z = scale * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        out.append((x + g).reshape(-1))
    return out


def _exact_newton(case, seed):
    cells, k = _cells(case), case["degree"]
    sizes = tuple(100.0 * c / max(cells) for c in cells)
    L = _Lattice(cells, sizes, k)
    u = _grains(cells, sizes, k, np.random.default_rng(seed))
    dt, m, kappa = 0.5, 1.0, 2.0
    for _ in range(1 + case["increments"]):
        old = L.split(u)
        for _ in range(12):
            v = L.split(u)
            r = L.integrate(old - v - dt * m * 4.0 * v * (v - 1.0) * (v - 0.5),
                            [-dt * kappa * m * g for g in L.grad(v)])
            if (r / L.mass).abs().max() < 1e-15:
                break
            f = 1.0 + dt * m * (12.0 * v * (v - 1.0) + 2.0)

            def A(d):
                w = L.split(d)
                return L.integrate(f * w, [dt * kappa * m * g for g in L.grad(w)])

            x, z = torch.zeros_like(r), r / L.mass
            p, rz = z.clone(), (r * z).sum()
            stop = 1e-28 * rz
            for _ in range(400):
                q = A(p)
                a = rz / (p * q).sum()
                x += a * p
                r = r - a * q
                z = r / L.mass
                new = (r * z).sum()
                if new < stop:
                    break
                p = z + (new / rz) * p
                rz = new
            u = u + x
    return [u.reshape(-1)]


def _exact_ensemble(case, seed):
    meshes, mw, ka, ics, dt = _ensemble(case, seed)
    out = []
    for m, a, b, u in zip(meshes, mw, ka, ics):
        L = _Lattice(tuple(m.subdivisions[:2]), (100.0, 100.0), m.degree)
        for _ in range(case["steps"]):
            u = _allen_cahn_step(L, u, dt, float(a), float(b))
        out.append(u.reshape(-1))
    return out


def _acch_step(L, c, n, dt, Mc, Mn, Kn):
    cv, nv = L.split(c), L.split(n)
    cx, nx = L.grad(cv), L.grad(nv)
    fa = -1.6704 - 4.776 * cv + 5.1622 * cv ** 2 - 2.7375 * cv ** 3 + 1.3687 * cv ** 4
    fa_c = -4.776 + 2 * 5.1622 * cv - 3 * 2.7375 * cv ** 2 + 4 * 1.3687 * cv ** 3
    fa_cc = 2 * 5.1622 - 6 * 2.7375 * cv + 12 * 1.3687 * cv ** 2
    fb = -1.5924 - 5.9746 * cv + 5.0 * cv ** 2
    fb_c = -5.9746 + 10.0 * cv
    h = 10.0 * nv ** 3 - 15.0 * nv ** 4 + 6.0 * nv ** 5
    hn = 30.0 * nv ** 2 - 60.0 * nv ** 3 + 30.0 * nv ** 4
    A, B = (1.0 - h) * fa_cc + h * 10.0, (fb_c - fa_c) * hn
    c1 = L.integrate(cv, [-dt * Mc * (A * g + B * q) for g, q in zip(cx, nx)]) / L.mass
    n1 = L.integrate(nv - dt * Mn * (fb - fa) * hn, [-dt * Kn * Mn * q for q in nx]) / L.mass
    return c1, n1


def _exact_adjoint(case, seed):
    cells, sizes, c0, n0, dt, consts = _acch(case, seed)
    L = _Lattice(cells, sizes, case["degree"])
    c0, n0 = c0.clone().requires_grad_(), n0.clone().requires_grad_()
    par = torch.tensor([consts[0], consts[2]], dtype=torch.float64, device=DEV, requires_grad=True)
    c, n = c0, n0
    for _ in range(case["steps"]):
        c, n = _acch_step(L, c, n, dt, par[0], consts[1], par[1])
    w = torch.from_numpy(_adjoint_weights(c0.numel(), seed)).to(DEV)
    J = (c.reshape(-1) * w[: c.numel()]).sum() + (n.reshape(-1) * w[c.numel():]).sum()
    J.backward()
    du0 = torch.cat([c0.grad.reshape(-1), n0.grad.reshape(-1)])
    return {"params": par.grad, "du0": du0, "c": c.detach().reshape(-1), "n": n.detach().reshape(-1)}
