"""A cell launch that fails (an error code from a stand-in for the operator's launch function, nothing
reaches the GPU) leaves the handle usable: the call reports the error, and the same call repeated gives
what an undisturbed handle gives, also where the failure came in the middle of a graph capture."""
import ctypes as C

import numpy as np
import pytest

from phasefield_gb300 import capi
from phasefield_gb300 import workloads as W

pytestmark = pytest.mark.gpu

LAUNCH = C.CFUNCTYPE(C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p)


class ModelOps(C.Structure):
    _fields_ = [("name", C.c_char_p), ("has_lhs", C.c_bool), ("make_object", C.c_void_p), ("launch", LAUNCH)]


class Stand_in:
    """A model registered under another name whose launches pass through until the n-th."""
    kept = []

    def __init__(self, lib, model):
        find = lib._ZN3ppf10find_modelEPKc
        find.restype, find.argtypes = C.POINTER(ModelOps), [C.c_char_p]
        real = find(model.encode()).contents
        self.calls, self.fail_at, self.real = 0, None, real.launch

        def launch(*a):
            self.calls += 1
            if self.calls == self.fail_at:
                return 1  # cudaErrorInvalidValue
            return self.real(*a)

        self.name = "%s_stand_in_%d" % (model, len(Stand_in.kept))
        self.ops = ModelOps(self.name.encode(), real.has_lhs, real.make_object, LAUNCH(launch))
        Stand_in.kept.append(self)  # (the registry keeps a pointer)
        register = lib._ZN3ppf14register_modelEPKNS_8ModelOpsE
        register.restype, register.argtypes = None, [C.POINTER(ModelOps)]
        register(C.byref(self.ops))


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("make,fields", [
    (lambda: W.coupled_acch_2d(refine=3, degree=2, size=32.0, dt=1e-3, n_precip=3), (0, 1)),
    (lambda: W.cahn_hilliard_3d(refine=2, degree=1, size=4.0, dt=1e-5), (0, 1)),
])
def test_explicit_run(gpu_lib, monkeypatch, make, fields):
    monkeypatch.setenv("PPF_CONTRACTION_MODE", "1")  # (no timing launches)
    n = 23

    def run(fail_at):
        wl = make()
        s = Stand_in(gpu_lib, wl.model)
        wl.model = s.name
        p = wl.make_problem()
        s.fail_at = fail_at
        if fail_at:
            with pytest.raises(capi.PPFError):
                p.solve(n)
        p.solve(n)
        assert p.get_time()[0] == n + 1
        out = [p.download_solution(f) for f in fields]
        p.close()
        return out, s.calls

    ref, total = run(None)
    for fail_at in range(1, total + 1):
        for got, r, f in zip(run(fail_at)[0], ref, fields):
            assert rel_l2(got, r) < 1e-12, (fail_at, f)


@pytest.mark.parametrize("mixed", [0, 1])
def test_multigrid_solve(gpu_lib, monkeypatch, mixed):
    monkeypatch.setenv("PPF_CONTRACTION_MODE", "1")
    prm = dict(tolerance_type=1, tolerance=1e-10, max_iterations=200, preconditioner=2, mg_depth=3, smoother_degree=4,
               mixed_precision=mixed)

    def solved(fail_at):
        wl = W.eshelby_3d(refine=2, degree=1, size=16.0, n_incl=5)
        s = Stand_in(gpu_lib, wl.model)
        wl.model = s.name
        p = wl.make_problem()
        p.set_linear_params(0, **prm)
        s.fail_at = fail_at
        diagonal = None
        if fail_at:
            with pytest.raises(capi.PPFError):
                p.linear_solve(0)
            if not mixed:
                diagonal = p.lhs_diagonal(0)
        its, _ = p.linear_solve(0)
        if diagonal is None and not mixed:
            diagonal = p.lhs_diagonal(0)
        out = its, p.download(0), diagonal, s.calls
        p.close()
        return out

    its, ref, diagonal, total = solved(None)
    for fail_at in range(1, total - (not mixed) + 1):
        its2, u, d, _ = solved(fail_at)
        assert its2 <= its + 1, fail_at
        assert rel_l2(u, ref) < 1e-8, fail_at
        if not mixed:
            assert rel_l2(d, diagonal) < 1e-12, fail_at
