"""The lane kernel's conversions (include/prismspf/gpu/fixed_point.cuh: to_fixed_cut,
to_fixed_cut_scaled, to_double_cut) against exact rational arithmetic on the CPU, at the ends of the
ranges their callers guarantee: block exponents from EXP_FLOOR up, scales within 2^+-60, one-word and
two-word integers, zeros, negated results and results beyond the normal range."""
import ctypes as C
import math
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
ONE = 1 << 63

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def lc(tmp_path_factory):
    out = tmp_path_factory.mktemp("lane_shim") / "liblane_shim.so"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "include"),
                        str(ROOT / "tests" / "lane_conversions_shim.cc"), "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(out))
    lib.lcs_to_fixed.restype = C.c_longlong
    lib.lcs_to_fixed.argtypes = [C.c_double, C.c_int]
    lib.lcs_to_fixed_scaled.restype = C.c_longlong
    lib.lcs_to_fixed_scaled.argtypes = [C.c_double, C.c_int, C.c_ulonglong, C.c_int]
    lib.lcs_to_double.restype = C.c_double
    lib.lcs_to_double.argtypes = [C.c_longlong, C.c_int, C.c_ulonglong, C.c_int, C.c_int, C.c_int, C.c_uint]
    lib.lcs_scale.argtypes = [C.c_double, C.POINTER(C.c_ulonglong), C.POINTER(C.c_int)]
    return lib


def scale(lc, s):
    sig, k = C.c_ulonglong(), C.c_int()
    lc.lcs_scale(s, C.byref(sig), C.byref(k))
    return sig.value, k.value


def cut(q):
    """A rational rounded towards zero."""
    n = abs(q).__floor__()
    return -n if q < 0 else n


@pytest.mark.parametrize("E", [192, 1023, 2046])
def test_to_fixed_cuts_towards_zero(lc, E):
    rng = np.random.default_rng(E)
    top = lc.lcs_top_values()
    for drop in list(range(0, 66)) + [100]:
        for _ in range(8):
            e = E - drop
            v = math.ldexp(float(rng.uniform(1.0, 2.0)), e - 1023) * (1 if rng.random() < 0.5 else -1)
            want = cut(Fraction(v) * Fraction(2) ** (1023 + top - E))
            assert lc.lcs_to_fixed(v, E) == want, (v, E)
            assert abs(want) < 2 ** (top + 1)
    for v in (0.0, -0.0, 5e-324, -2.0 ** -1023):
        assert lc.lcs_to_fixed(v, E) == 0


@pytest.mark.parametrize("s", [1.5, 0.08, 3.0, 1.0 / 216.0, 1.0, 2.0 ** 59 * 1.9, 2.0 ** -60])
def test_to_fixed_scaled_is_less_than_a_unit_off(lc, s):
    rng = np.random.default_rng(7)
    top = lc.lcs_top_integral()
    sig, k = scale(lc, s)
    for _ in range(400):
        e = int(rng.integers(260, 1900))
        v = math.ldexp(float(rng.uniform(1.0, 2.0)), e - 1023) * (1 if rng.random() < 0.5 else -1)
        E = max(192, e + k + 1 + int(rng.integers(0, 70)))
        exact = Fraction(v) * Fraction(sig, ONE) * Fraction(2) ** (k + 1023 + top - E)
        got = lc.lcs_to_fixed_scaled(v, E, sig, k)
        assert 0 <= abs(exact) - abs(got) < 1 and (got == 0 or (got < 0) == (v < 0)), (v, E, s)
    for E in (192, 600):
        assert lc.lcs_to_fixed_scaled(0.0, E, sig, k) == 0


def nearest(q):
    """A rational in double's normal range rounded to nearest, ties away from zero."""
    if q == 0:
        return 0.0
    a = abs(q)
    e = 0
    while Fraction(2) ** e > a:
        e -= 1
    while Fraction(2) ** (e + 1) <= a:
        e += 1
    m = a / Fraction(2) ** (e - 52)
    n = m.__floor__()
    if m - n >= Fraction(1, 2):
        n += 1
    return math.copysign(math.ldexp(float(n), e - 52), -1.0 if q < 0 else 1.0)


@pytest.mark.parametrize("lsb", [-890, -59, 0, 700])
def test_to_double_rounds_to_nearest(lc, lsb):
    rng = np.random.default_rng(11)
    xs = [0, 1, -1, 2 ** 31, 2 ** 32 - 1, 2 ** 32, 2 ** 53 + 1, -(2 ** 53 + 1), 2 ** 54 - 1, 2 ** 63 - 1, -(2 ** 63 - 1)]
    xs += [int(rng.integers(1, 2 ** 62)) >> int(rng.integers(0, 62)) for _ in range(400)]
    for x in xs:
        for s in (1, -1):
            want = nearest(Fraction(s * x) * Fraction(2) ** lsb)
            assert lc.lcs_to_double(s * x, lsb, ONE, 0, 0, 0, 0) == want, (x, lsb)
            assert lc.lcs_to_double(s * x, lsb, ONE, 0, 1, 0, 0) == want
            assert lc.lcs_to_double(s * x, lsb, ONE, 0, 0, 0, 0x80000000) == -want


@pytest.mark.parametrize("s", [1.25, 1.0 / 27.0, 1.999999])
def test_to_double_scaled_is_half_a_last_place_and_two_units_off(lc, s):
    rng = np.random.default_rng(13)
    sig, k = scale(lc, s)
    for _ in range(600):
        x = int(rng.integers(-2 ** 62, 2 ** 62)) >> int(rng.integers(0, 60))
        lsb = int(rng.integers(-300, 300))
        exact = Fraction(x) * Fraction(2) ** lsb * Fraction(sig, ONE)
        got = lc.lcs_to_double(x, lsb, sig, 1, 0, 0, 0)
        ulp = Fraction(math.ulp(got)) if got else Fraction(0)
        assert abs(Fraction(got) - exact) <= ulp / 2 + 2 * Fraction(2) ** lsb, (x, lsb, s)


def test_to_double_beyond_the_range_and_of_a_bad_cell(lc):
    big = 2 ** 62 + 12345
    assert not math.isfinite(lc.lcs_to_double(big, 1000, ONE, 0, 1, 0, 0))
    assert not math.isfinite(lc.lcs_to_double(-big, 1000, ONE, 0, 1, 0, 0))
    for x in (0, 1, -big):
        assert math.isnan(lc.lcs_to_double(x, 1000, ONE, 0, 1, 1, 0))
