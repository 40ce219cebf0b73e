"""Device memory of a run: the second accumulator of explicit solves is the solved fields' only."""
import pytest

from phasefield_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_graphs_need_no_memory_for_fields_they_do_not_solve(gpu_lib):
    import torch

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    W.allen_cahn_2d(refine=4, degree=1).make_problem().solve(60)  # (the kernels' own memory)
    p = W.allen_cahn_2d(refine=10, degree=1, dt=1e-5).make_problem()  # n, and two fields of post-processing
    p.solve(1)
    before, field = used(), 8 * p.field_length(0)
    p.solve(60)
    assert used() - before < field, "a graph of increments allocated vectors"
    p.close()
