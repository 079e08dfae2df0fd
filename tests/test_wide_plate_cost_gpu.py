"""Plates of more than 1024 columns, whose rows have more words than a warp has
lanes: the same packing costs little more there than on plates just below that
width, and comes out as the oracle's."""
import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem
from oracle import oracle_decode

pytestmark = pytest.mark.gpu


def _decoder(width, P):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import DeviceDecoder
    inst = instances.make_instance("w", 60, [(200, width), (300, width)], 3, bbox_min=20, bbox_max=100)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    return torch, pk, DeviceDecoder(pk, max_pop=P, pool_bins=8 * P * pk.n_machines)


def _best_ms(torch, dec, chrom):
    best = float("inf")
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        dec.decode(chrom, kernel_events=e)
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best


def test_cost_does_not_jump_past_a_warps_words():
    P = 2000
    ms = []
    for width in (1024, 1280):
        torch, pk, dec = _decoder(width, P)
        ms.append(_best_ms(torch, dec, torch.from_numpy(instances.chromosomes(P, pk.n_genes, 7)).cuda()))
    # 1.25 times the columns; the search itself stops at the first fit, so up to twice the time is width
    assert ms[1] < 2.0 * ms[0], ms


@pytest.mark.parametrize("width", [1025, 1280, 1984, 2049])
def test_matches_oracle(width):
    torch, pk, dec = _decoder(width, 24)
    ch = instances.chromosomes(24, pk.n_genes, 9)
    ref, rlog = oracle_decode(pk, ch, n_threads=8, with_log=True)
    log = torch.full((24, pk.n_machines, pk.n_genes, 5), -7, dtype=torch.int32, device="cuda")
    out = dec.decode(torch.from_numpy(ch).cuda(), log=log)
    torch.cuda.synchronize()
    assert int(dec.status.item()) == abi.OK
    got = log.cpu().numpy().reshape(-1).view(abi.PLACEMENT_DTYPE).reshape(rlog.shape)
    assert np.array_equal(out.cpu().numpy(), ref)
    assert (got == rlog).all()
