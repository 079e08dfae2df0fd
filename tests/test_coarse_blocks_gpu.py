"""The coarse test's kernel paths against the oracle, makespans and placements:
both block heights, plates whose rows do not fill the last block and whose
columns end around a word, a plate wider than a warp's words, items whose CTAs
reuse the plates of earlier ones, in every launch shape."""
import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem
from oracle import oracle_decode

pytestmark = pytest.mark.gpu

# (parts, plates, mask sides, chromosomes)
CASES = {
    "small_masks_ragged_rows": (30, [(61, 65), (33, 96)], (3, 20), 64),         # blocks of four rows
    "filled_plates": (60, [(90, 97), (75, 130)], (8, 44), 64),                  # blocks of four rows
    "tall_masks": (24, [(131, 127), (150, 64)], (48, 62), 64),                  # blocks of eight rows
    "wide_plate": (40, [(45, 1100), (60, 1024)], (20, 40), 32),                 # more words a row than lanes
    "many_items": (12, [(70, 70), (40, 111), (63, 33)], (10, 30), 3000),        # several items per CTA
}
SHAPES = [(0, 0, -1, -1), (4, 0, 1, -1), (4, 2, 0, 3), (2, 0, -1, -1), (2, 4, 1, 0), (1, 0, -1, -1)]


@pytest.mark.parametrize("name", list(CASES))
def test_matches_oracle(name):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import DeviceDecoder
    n, plates, (lo, hi), P = CASES[name]
    inst = instances.make_instance(name, n, plates, 3, bbox_min=lo, bbox_max=hi, scale_machines=True)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    ch = instances.chromosomes(P, n, 11)
    ref, rlog = oracle_decode(pk, ch, n_threads=8, with_log=True)
    dec = DeviceDecoder(pk, max_pop=P, pool_bins=8 * P * pk.n_machines)  # up to eight plates per item, whatever the shape
    chrom = torch.from_numpy(ch).cuda()
    for shape in SHAPES:
        dec.set_launch_config(*shape)
        log = torch.full((P, pk.n_machines, n, 5), -7, dtype=torch.int32, device="cuda")
        for _ in range(2):  # the second launch finds the first one's plates in the workspace
            out = dec.decode(chrom, log=log)
        torch.cuda.synchronize()
        assert int(dec.status.item()) == 0, shape
        np.testing.assert_array_equal(out.cpu().numpy(), ref, err_msg=str(shape))
        got = log.cpu().numpy().reshape(-1).view(abi.PLACEMENT_DTYPE).reshape(rlog.shape)
        assert (got == rlog).all(), shape
