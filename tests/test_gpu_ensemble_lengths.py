"""Ensemble runs of every length after each other, from every phase of the accumulator rotation, replayed
from graphs of one and of several rotations, against plain launches (1e-12 relative L2: the order of the
scatter's FP64 additions), also where the tile shape changes in between."""
import numpy as np
import pytest

from phasefield_gb300 import ensemble as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs", [(3, 100, 9, 30, 3), (100, 10, 17, 10, 100), (1, 2, 150, 1, 24, 23, 25), (9,) * 14])
@pytest.mark.parametrize("tune", [False, True])
def test_runs_after_each_other(gpu_lib, runs, tune):
    meshes, mw, ka, ics = E.allen_cahn_ensemble(n_instances=5, min_cells=8, max_cells=24, seed=3)
    res = []
    for use_graph in (False, True):
        ens = E.Ensemble(meshes, mw, ka, 0.01)
        for i, ic in enumerate(ics):
            ens.upload(i, ic)
        out = []
        for k, n in enumerate(runs):
            if tune and k == 2:
                ens.autotune(steps=1)
            ens.run(n, use_graph=use_graph)
            out += [ens.download(i) for i in range(len(meshes))]
        res.append(out)
    for a, b in zip(*res):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(a)
