"""The lane kernel's conversions at the ends of the normal range (include/prismspf/gpu/fixed_point.cuh)
against exact arithmetic, on the CPU."""
import ctypes as C
import math
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
ONE = 1 << 63

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def lc(tmp_path_factory):
    d = tmp_path_factory.mktemp("lane_ranges")
    src = d / "shim.cc"
    src.write_text("""#include <prismspf/gpu/fixed_point.cuh>
namespace fx = prismspf::gpu::fx;
extern "C" {
double to_double(long long x, int lsb, unsigned long long sig, int scaled, int wide, int bad) {
  return fx::to_double_cut(x, lsb, sig, scaled != 0, wide != 0, bad != 0);
}
int lane_floor(int up, int down) { return fx::lane_floor(up, down); }
long long to_fixed(double v, int E) { return fx::to_fixed_cut<fx::LANE_TOP_VALUES>(v, fx::high_exponent(E)); }
long long to_fixed_scaled(double v, int E, unsigned long long sig, int k, int q1) {
  return q1 ? fx::to_fixed_cut_scaled<fx::LANE_TOP_INTEGRAL_Q1>(v, fx::high_exponent(E), sig, k)
            : fx::to_fixed_cut_scaled<fx::LANE_TOP_INTEGRAL>(v, fx::high_exponent(E), sig, k);
}
}
""")
    out = d / "shim.so"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "include"), str(src), "-o",
                        str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(out))
    lib.to_double.restype = C.c_double
    lib.to_double.argtypes = [C.c_longlong, C.c_int, C.c_ulonglong, C.c_int, C.c_int, C.c_int]
    lib.to_fixed.restype = lib.to_fixed_scaled.restype = C.c_longlong
    lib.to_fixed.argtypes = [C.c_double, C.c_int]
    lib.to_fixed_scaled.argtypes = [C.c_double, C.c_int, C.c_ulonglong, C.c_int, C.c_int]
    return lib


def test_results_at_the_upper_end(lc):
    """Rounding up to the next power of two at or above the range gives an infinity of the sum's sign."""
    assert lc.to_double(1 << 62, 961, ONE, 0, 1, 0) == 2.0 ** 1023
    largest = math.ldexp(float((1 << 53) - 1), 971)
    assert lc.to_double(((1 << 53) - 1) << 9, 962, ONE, 0, 1, 0) == largest
    for lsb in (962, 963, 1500, 2900):
        for x in ((1 << 62) - 1, (1 << 62) + 12345, (1 << 63) - 1):
            assert lc.to_double(x, lsb, ONE, 0, 1, 0) == math.inf, (x, lsb)
            assert lc.to_double(-x, lsb, ONE, 0, 1, 0) == -math.inf, (x, lsb)
    assert math.isnan(lc.to_double((1 << 62) - 1, lsb, ONE, 0, 1, 1))


@pytest.mark.parametrize("scaled", [0, 1])
def test_results_below_the_normal_range_are_signed_zeros(lc, scaled):
    """One-word sums (what a cell at the floor leaves of its smallest values) down to nothing."""
    for x in (3, -3, (1 << 31) + 1, -(1 << 31)):
        for lsb in (-1200, -1400, -3000):
            got = lc.to_double(x, lsb, ONE, scaled, 0, 0)
            assert got == 0.0 and math.copysign(1.0, got) == math.copysign(1.0, x), (x, lsb)
    # the smallest normal number, and the next power of two below it
    assert lc.to_double(1 << 31, -1053, ONE, 0, 0, 0) == 2.0 ** -1022
    assert lc.to_double(1 << 31, -1054, ONE, 0, 0, 0) == 0.0


@pytest.mark.parametrize("down", [-60, -33, -1, 0, 60])
def test_two_word_sums_at_the_floor_are_normal(lc, down):
    """The least sum of more than 32 bits, scaled by 2^down, in a cell at its floor."""
    for top in (57, 59):
        lsb = lc.lane_floor(0, down) - 1023 - top + down
        for s in (1, -1):
            assert lc.to_double(s << 32, lsb, ONE, 0, 0, 0) == s * math.ldexp(1.0, 32 + lsb) != 0.0
            assert lc.to_double(s << 33, lsb, ONE, 1, 0, 0) == s * math.ldexp(1.0, 33 + lsb) != 0.0


def test_zeros_shift_out_at_the_floor(lc):
    """From the least block exponent on (a positive scale's exponent more) zeros and subnormals give 0,
    and the smallest block keeps its bits."""
    E = lc.lane_floor(0, 0)
    assert E <= 64
    for v in (0.0, -0.0, 5e-324, -2.0 ** -1023):
        assert lc.to_fixed(v, E) == 0
        for k in (-60, -1, 0, 1, 60):
            for sig in (ONE, ONE + 12345, 2 * ONE - 1):
                for q1 in (0, 1):
                    assert lc.to_fixed_scaled(v, lc.lane_floor(k, 0), sig, k, q1) == 0, (v, k)
    for m in (1.0, 1.5, 2.0 - 2.0 ** -52):
        assert lc.to_fixed(math.ldexp(m, E - 1023), E) == int(math.ldexp(m, 52)) << 7
        assert lc.to_fixed(math.ldexp(-m, E - 1023 - 40), E) == -(int(math.ldexp(m, 52)) << 7 >> 40)
