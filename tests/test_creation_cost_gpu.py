"""Device memory of a problem whose masks have many short runs: the runs are
their own pieces, so they are kept once."""
import numpy as np
import pytest

from brkga_fft2_b200 import pack_problem
from tests import edge_shapes

pytestmark = pytest.mark.gpu


def test_short_runs_are_kept_once():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import _NativeProblem
    masks = [edge_shapes.checker(700, 600 + 4 * k, 2) for k in range(12)]
    inst = edge_shapes.build("runs", [(1000, 1000)], masks, 1)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    runs = sum(int((np.diff(np.pad(np.rot90(m, r), ((0, 0), (1, 0))).astype(np.int8), axis=1) == 1).sum())
               for m in masks for r in range(4))
    _NativeProblem(pk).close()  # loads the kernels
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    native = _NativeProblem(pk)
    taken = before - torch.cuda.mem_get_info()[0]
    native.close()
    # eight bytes a run, the bit masks, the row filter and allocation granularity; twice the runs would be 16 bytes
    assert 8 * runs > 30 << 20
    assert taken < 8 * runs + (12 << 20), (taken, runs)
