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
}
""")
    out = d / "shim.so"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "include"), str(src), "-o",
                        str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(out))
    lib.to_double.restype = C.c_double
    lib.to_double.argtypes = [C.c_longlong, C.c_int, C.c_ulonglong, C.c_int, C.c_int, C.c_int]
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
