"""Inserting masks whose rows end around the words at which the insertion
changes its path (four and eight words a row), against the oracle."""
import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem
from oracle import oracle_decode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(31, 34), (95, 98), (127, 130), (159, 162), (255, 258), (287, 290)])
def test_matches_oracle(lo, hi):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import DeviceDecoder
    n, P = 10, 24
    inst = instances.make_instance("widths", n, [(2 * hi + 5, 2 * hi + 33), (hi + 9, 3 * hi)], lo, bbox_min=lo,
                                   bbox_max=hi, scale_machines=True)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    ch = instances.chromosomes(P, n, 17)
    ref, rlog = oracle_decode(pk, ch, n_threads=8, with_log=True)
    dec = DeviceDecoder(pk, max_pop=P, pool_bins=n * P * pk.n_machines)
    log = torch.full((P, pk.n_machines, n, 5), -7, dtype=torch.int32, device="cuda")
    out = dec.decode(torch.from_numpy(ch).cuda(), log=log)
    torch.cuda.synchronize()
    assert int(dec.status.item()) == 0
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    got = log.cpu().numpy().reshape(-1).view(abi.PLACEMENT_DTYPE).reshape(rlog.shape)
    assert (got == rlog).all()
