"""brkga_decode_noalloc on plates whose erosion planes are as large as their grids
(blocks of four rows): against the workspace decode, and with as many plates as
the 64 MiB array has grids for."""
import ctypes

import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem
from tests import edge_shapes

pytestmark = pytest.mark.gpu


def _both(inst, P, per_item, seed):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import DeviceDecoder
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    dd = DeviceDecoder(pk, max_pop=P, pool_bins=per_item * P * pk.n_machines)
    chrom = torch.from_numpy(instances.chromosomes(P, pk.n_genes, seed)).cuda()
    shape = (P, pk.n_machines, pk.n_genes, 5)
    ref_log = torch.full(shape, -7, dtype=torch.int32, device="cuda")
    ref = dd.decode(chrom, log=ref_log)
    out = torch.full((P,), -1.0, dtype=torch.float64, device="cuda")
    log = torch.full(shape, -7, dtype=torch.int32, device="cuda")
    status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    assert dd.lib.brkga_decode_noalloc(dd.native.handle, ctypes.c_void_p(chrom.data_ptr()), P,
                                       ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(log.data_ptr()),
                                       ctypes.c_void_p(status.data_ptr()),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == abi.OK
    torch.cuda.synchronize()
    assert int(dd.status.item()) == abi.OK
    assert int(status.item()) == abi.OK
    assert torch.equal(out, ref)
    assert torch.equal(log, ref_log)
    return dd.counters()[2]


@pytest.mark.parametrize("plates,sides", [([(200, 200)] * 2, (14, 25)), ([(61, 97), (90, 70)], (14, 25))])
def test_blocks_of_four_rows(plates, sides):
    inst = instances.make_instance("n", 60, plates, 5, bbox_min=sides[0], bbox_max=sides[1])
    for seed in (1, 2):  # the second call finds the first one's plates in the arrays
        _both(inst, 120, 16, seed)


@pytest.mark.parametrize("rows,width,parts", [(1, 8160, 30), (3, 8160, 14), (13, 3776, 12), (15, 3264, 12), (18, 2720, 12)])
def test_pool_is_not_limited_by_the_planes(rows, width, parts):
    """Parts of a whole plate each for 1,184 resident CTAs with four plates of
    their own; what is beyond those, 30,800 pool plates of one row or 9,500 of 13,
    is up to 0.95 of what the 64 MiB hold grids of."""
    inst = edge_shapes.build("full", [(rows, width)], [np.ones((rows, width), np.uint8) for _ in range(parts)], 3)
    assert _both(inst, 1184, parts, 3) == parts * 1184
