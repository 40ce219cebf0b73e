"""Shared memory of the cell kernels' launches: the tables a kernel stages hold nothing of the lane
kernel's, so adaptive meshes of many levels fit the 227 KB of a block. Host code, compiled with nvcc."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(not Path(NVCC).exists(), reason="needs nvcc")

LIMIT = 232448


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    d = tmp_path_factory.mktemp("smem")
    (d / "main.cu").write_text("""#include <prismspf/gpu/amr_cell_kernel.cuh>
#include <prismspf/gpu/cell_kernel.cuh>
#include <cstdio>
int main() {
  for (int levels : {1, 6, 13, 14, 15, 16})
    for (int in : {1, 21, 22, 23, 24})
      for (int out : {4, 44, 48})
        std::printf("%d %d %d %zu\\n", levels, in, out, ppf::amr_cell_smem_bytes<3, 2, double>(levels, in, out));
}
""")
    r = subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(ROOT / "include"), str(d / "main.cu"),
                        "-o", str(d / "main")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(d / "main")], capture_output=True, text=True, check=True).stdout
    return {tuple(map(int, line.split()[:3])): int(line.split()[3]) for line in out.splitlines()}


@pytest.mark.parametrize("levels,rows_in,rows_out", [(16, 21, 48), (15, 22, 48), (16, 22, 48), (16, 23, 44), (14, 23, 48),
                                                     (13, 24, 48)])
def test_many_levels_fit(sizes, levels, rows_in, rows_out):
    assert sizes[levels, rows_in, rows_out] <= LIMIT


def test_a_level_takes_little(sizes):
    assert (sizes[16, 1, 4] - sizes[6, 1, 4]) / 10 <= 3088  # (3568 with the lane kernel's members)
