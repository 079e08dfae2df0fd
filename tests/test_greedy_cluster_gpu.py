"""The greedy initial solution's cluster kernel at the sizes where its split
over CTAs and its state can go wrong, against the oracle: fewer plates than
CTAs, one plate more than a multiple of them, many plates of one machine, and
more parts than its shared-memory state holds."""
import numpy as np
import pytest

from brkga_fft2_b200 import instances, pack_problem
from oracle import oracle_initial_solution

pytestmark = pytest.mark.gpu

# (parts, plates, mask sides, times the gene list is repeated)
CASES = {
    "one_part": (1, [(40, 40)], (4, 20), 1),
    "one_plate": (12, [(200, 200)], (4, 20), 1),
    "three_machines": (40, [(60, 60), (64, 56), (90, 50)], (12, 40), 1),
    "plates_of_one_machine": (60, [(50, 50)], (20, 45), 1),
    "state_in_global_memory": (20, [(160, 160), (130, 170)], (3, 5), 420),
}


@pytest.mark.parametrize("name", list(CASES))
def test_greedy_matches_oracle(name):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import _NativeProblem
    from brkga_fft2_b200.initial import greedy_order, greedy_placements
    n, plates, (lo, hi), times = CASES[name]
    inst = instances.make_instance(name, n, plates, 5, bbox_min=lo, bbox_max=hi, scale_machines=True)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    order = np.repeat(greedy_order(inst.instance_parts, inst.heights, [float(m.sum()) for m in inst.masks]), times)
    machine, place, mk = greedy_placements(_NativeProblem(pk), order)
    ref_machine, ref_place, ref_mk = oracle_initial_solution(pk, order)
    np.testing.assert_array_equal(machine, ref_machine)
    assert (place == ref_place).all()
    np.testing.assert_array_equal(mk, ref_mk)
