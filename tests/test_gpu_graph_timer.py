"""The simulation time that callbacks read while increments are replayed from graphs, advanced on the
device: an application whose fields follow the time alone, against the closed form within 1e-12 (a few
hundred FP64 additions of terms of one sign), on a uniform and on an adaptive mesh, over run lengths that
take plain launches, graphs of one and of several periods and their ends."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
DT = 0.125


@pytest.fixture(scope="module")
def application(gpu_lib, tmp_path_factory):
    from phasefield_gb300 import app_build
    return app_build.compile_app(ROOT / "tests" / "dropin" / "timer", tmp_path_factory.mktemp("timer") / "timer")


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("steps,outputs", [(1, 1), (5, 1), (6, 2), (37, 1), (200, 1), (203, 7)])
def test_callbacks_read_the_time_of_their_increment(application, tmp_path, steps, outputs, adaptive):
    from test_gpu_dropin import read_vtu
    # (the criterion holds nowhere: one mesh, coarsened once if at all)
    extra = """
set mesh adaptivity = true
set remeshing period = 1000
set max refinement = 4
set min refinement = 3
subsection refinement criterion: 0
  set type = value
  set value lower bound = -10
  set value upper bound = -5
  set variables = n
end
""" if adaptive else ""
    (tmp_path / "parameters.prm").write_text(f"""
set global refinement = 4
subsection Rectangular mesh
  set x size = 16.0
  set y size = 16.0
end
set time step = {DT}
set number steps = {steps}
subsection output
  set number = {outputs}
end
{extra}""")
    r = subprocess.run([str(application), "-i", "parameters.prm"], cwd=tmp_path, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    files = sorted((tmp_path / "solutions").glob("solution_*.vtu"), key=lambda f: int(f.stem.split("_")[1]))
    assert int(files[-1].stem.split("_")[1]) == steps
    for f in files:
        k = int(f.stem.split("_")[1])
        if k == 0:
            continue
        n = sum(DT * (i * DT) * (1.0 + i / 1024.0) for i in range(1, k + 1))
        v = read_vtu(f)
        assert np.allclose(v["n"], n, rtol=1e-12, atol=0), (k, v["n"][0], n)
        assert np.allclose(v["m"], n + k * DT, rtol=1e-12, atol=0), k
