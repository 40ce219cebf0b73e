"""The choice of graphs for a loop of repeated periods (phasefield_gb300/csrc/graph_lengths.h), on the CPU."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("graph_lengths")
    (d / "shim.cc").write_text("""#include "graph_lengths.h"
extern "C" void choose(int periods, int one, long long replayed, int many, int* out) {
  const ppf::GraphChoice c = ppf::choose_graph(periods, one != 0, replayed, many);
  out[0] = c.capture;
  out[1] = c.replay;
}
""")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "phasefield_gb300" / "csrc"),
                        str(d / "shim.cc"), "-o", str(d / "shim.so")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(d / "shim.so"))
    lib.choose.argtypes = [C.c_int, C.c_int, C.c_longlong, C.c_int, C.POINTER(C.c_int)]

    def f(periods, one, replayed, many):
        out = (C.c_int * 2)()
        lib.choose(periods, int(one), replayed, many, out)
        return out[0], out[1]
    return f


class Loop:
    """The graphs a caller of choose_graph holds for one phase."""

    def __init__(self, choose):
        self.choose, self.one, self.replayed, self.many, self.recorded, self.launches = choose, False, 0, 0, 0, 0

    def run(self, periods):
        self.recorded = self.launches = 0
        while periods:
            capture, replay = self.choose(periods, self.one, self.replayed, self.many)
            assert 1 <= replay <= periods
            if capture:
                assert capture == replay
                self.recorded += capture
                if capture == 1:
                    assert not self.one
                    self.one = True
                else:
                    assert capture > self.many
                    self.many = capture
            assert self.one if replay == 1 else self.many == replay
            n = periods // replay
            self.launches += n
            if replay == 1:
                self.replayed += n
            periods -= n * replay


@pytest.mark.parametrize("first", [1, 5, 8, 31, 32, 50, 200])
def test_runs_of_any_length_after_any_other(choose, first):
    """Every period is replayed; a short first run does not keep later ones to short graphs."""
    loop = Loop(choose)
    loop.run(first)
    for n in (5, 8, 1, 50, 5, 50, 5, 1, 200):
        loop.run(n)
    for n in (1, 3, 5, 8, 50, 200):
        loop.run(n)
        assert loop.recorded == 0 and loop.launches == n // 8 + n % 8


def test_little_is_recorded_for_a_short_run(choose):
    for n in range(1, 32):
        loop = Loop(choose)
        loop.run(n)
        assert loop.recorded == 1 and loop.launches == n


def test_repeated_short_runs_become_one_graph(choose):
    loop = Loop(choose)
    for _ in range(7):
        loop.run(5)
    assert loop.many == 5
    loop.run(5)
    assert (loop.recorded, loop.launches) == (0, 1)
