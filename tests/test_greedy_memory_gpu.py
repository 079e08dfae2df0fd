"""The greedy's device memory: what a call of many large plates takes is given
back by it, what a small one takes stays with the problem, and later calls give
the same placements."""
import numpy as np
import pytest

from brkga_fft2_b200 import instances, pack_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plate,times,kept", [((3000, 3000), 15, False), ((300, 300), 1, True)])
def test_memory_after_a_call(plate, times, kept):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import _NativeProblem
    from brkga_fft2_b200.initial import greedy_order, greedy_placements
    inst = instances.make_instance("m", 20, [plate], 5, bbox_min=20, bbox_max=60)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    order = np.repeat(greedy_order(inst.instance_parts, inst.heights, [float(m.sum()) for m in inst.masks]), times)
    native = _NativeProblem(pk)
    greedy_placements(native, order[:1])  # loads the kernel
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    first = greedy_placements(native, order)
    taken = before - torch.cuda.mem_get_info()[0]
    # 300 plates of 3,000 rows x 96 words and their planes are 500 MB; the limit is 64 MiB
    assert taken <= 66 << 20
    small = greedy_placements(native, order[:5])
    again = greedy_placements(native, order)
    assert (first[0] == again[0]).all() and (first[1] == again[1]).all() and (first[2] == again[2]).all()
    assert (small[1] == first[1][:5]).all()
    if kept:  # nothing is allocated by a call that fits
        free = torch.cuda.mem_get_info()[0]
        greedy_placements(native, order)
        assert torch.cuda.mem_get_info()[0] == free
