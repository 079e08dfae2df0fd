"""The workspace of a launch of the default pool: a population of many items per
CTA needs no more than the cells of four plates an item and the tables, a smaller
population never more than a larger one, and the plates still suffice, also where
one machine's plates are much smaller than the others' and where all parts go to
one machine."""
import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 5, 20, 100, 148, 149, 300, 400, 444, 592, 600, 888, 889, 1000, 1184, 1185, 2000, 3000, 4000, 4736, 4737,
         6000, 9000, 9472, 9473, 12000, 16000, 30000, 60000]


def _problem(name):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import DeviceDecoder
    inst = {"p50m2": instances.p50m2, "p100m4": instances.p100m4, "p400m8": instances.p400m8,
            "small": lambda s: instances.make_instance("s", 60, [(61, 97), (90, 70)], 5, bbox_min=14, bbox_max=25)}[name](0)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    return torch, pk, DeviceDecoder(pk, max_pop=1)


@pytest.mark.parametrize("name", ["p50m2", "p100m4", "p400m8", "small"])
@pytest.mark.parametrize("shape", [(0, 0, -1, -1), (4, 0, -1, -1), (2, 0, 0, -1)])
def test_bytes(name, shape):
    torch, pk, dec = _problem(name)
    dec.set_launch_config(*shape)
    L, W = np.asarray(pk.arrays["bin_length"], np.int64), np.asarray(pk.arrays["bin_width"], np.int64)
    plate = int((L * (-(-W // 32) + 2)).max()) * 4 + 2 * int(L.max()) + 16  # rows of the cells' words and two more; 16 bits a row
    got = [dec.workspace_bytes(p) for p in SIZES]
    assert all(a <= b for a, b in zip(got, got[1:]))
    N, M = pk.n_genes, pk.n_machines
    for p, b in zip(SIZES, got):
        items = p * M
        if items < 16 * 4736:  # fewer than sixteen items per CTA of the shape of most CTAs
            continue
        tables = items * (2 * N + 16) + 16 * p + 4736 * N * 48 + (1 << 20)
        assert b <= 4 * items * plate + tables, p


def _uneven_plates():
    return instances.make_instance("u", 64, [(120, 120)] * 7 + [(36, 36)], 5, bbox_min=18, bbox_max=34)


@pytest.mark.parametrize("name,P,one_machine", [("p100m4", 6000, False), ("p100m4", 6000, True), ("small", 6000, False),
                                                ("uneven", 6000, False), ("uneven", 4000, True)])
def test_default_pool_serves_many_waves(name, P, one_machine):
    import torch
    from brkga_fft2_b200.evaluator import DeviceDecoder
    if name == "uneven":
        inst = _uneven_plates()
        pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    else:
        torch, pk, _ = _problem(name)
    keys = instances.chromosomes(P, pk.n_genes, 3)
    if one_machine:  # the first machine's interval, which is what a population may settle on
        keys[:, pk.n_genes:] *= 0.999 / pk.n_machines
    dec = DeviceDecoder(pk, max_pop=P)
    ample = DeviceDecoder(pk, max_pop=P, pool_bins=max(8 * P * pk.n_machines, 40 * P))
    chrom = torch.from_numpy(keys).cuda()
    out, ref = dec.decode(chrom), ample.decode(chrom)
    torch.cuda.synchronize()
    assert int(ample.status.item()) == abi.OK
    assert int(dec.status.item()) == abi.OK
    assert torch.equal(out, ref)
