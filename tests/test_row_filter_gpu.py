"""Parts whose rows share no wide run of columns (lattices, plates with holes,
thin and small parts): their test is by rows instead of blocks of rows.  It costs
little more than the test of solid parts that pack alike, and every form of it
gives the oracle's makespans and placements."""
import numpy as np
import pytest

from brkga_fft2_b200 import abi, instances, pack_problem
from oracle import oracle_decode
from tests import edge_shapes

pytestmark = pytest.mark.gpu


def lattice(h, w, pitch, bar=1):
    m = np.zeros((h, w), np.uint8)
    m[np.arange(h) % pitch < bar] = 1
    m[:, np.arange(w) % pitch < bar] = 1
    m[-1] = 1
    m[:, -1] = 1
    return m


def _side(rng, lo, hi):
    return int(rng.integers(lo, hi + 1))


def _packed(n, plates, make, seed=1):
    rng = np.random.default_rng(seed)
    inst = edge_shapes.build("rows", plates, [make(rng) for _ in range(n)], seed)
    return pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)


def _decoder(pk, P):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200.evaluator import DeviceDecoder
    return torch, DeviceDecoder(pk, max_pop=P, pool_bins=16 * P * pk.n_machines)


def _best_ms(pk, P):
    torch, dec = _decoder(pk, P)
    chrom = torch.from_numpy(instances.chromosomes(P, pk.n_genes, 5)).cuda()
    best = float("inf")
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        dec.decode(chrom, kernel_events=e)
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best


@pytest.mark.parametrize("pitch,bar", [((5, 9), 1), ((12, 20), 5)])
def test_lattices_cost_little_more_than_solid_parts(pitch, bar):
    """No part fits into another's holes, so both sets pack the same way."""
    P, plates = 2000, [(300, 300)] * 3
    hollow = _packed(60, plates, lambda r: lattice(_side(r, 30, 90), _side(r, 30, 90), _side(r, *pitch), bar))
    solid = _packed(60, plates, lambda r: np.ones(lattice(_side(r, 30, 90), _side(r, 30, 90), _side(r, *pitch)).shape, np.uint8))
    ms = _best_ms(hollow, P), _best_ms(solid, P)
    assert ms[0] < 2.0 * ms[1], ms


# (parts, plates, mask of one part, chromosomes)
CASES = {
    "lattices": (24, [(90, 97), (100, 64)], lambda r: lattice(_side(r, 8, 50), _side(r, 8, 50), _side(r, 3, 9)), 64),
    "thin": (40, [(61, 65), (64, 96)], lambda r: np.ones((_side(r, 1, 3), _side(r, 1, 60)), np.uint8), 64),
    "small": (60, [(33, 31), (20, 129)], lambda r: edge_shapes.random_blob(r, _side(r, 1, 6), _side(r, 1, 6)), 64),
    "few_plates_many_items": (16, [(25, 25), (19, 40), (40, 33)], lambda r: np.ones((_side(r, 1, 12), _side(r, 1, 12)), np.uint8), 3000),
    "filter_rows": (20, [(140, 140), (150, 161)], lambda r: lattice(_side(r, 62, 130), _side(r, 5, 60), 4), 48),  # more rows than the filter holds
    "wide_plate": (24, [(45, 1100), (60, 1024)], lambda r: lattice(_side(r, 5, 40), _side(r, 5, 300), _side(r, 3, 9)), 32),
    "mixed": (40, [(90, 130), (120, 97)], lambda r: lattice(_side(r, 20, 60), _side(r, 20, 60), 5) if r.random() < 0.3
              else np.ones((_side(r, 20, 60), _side(r, 20, 60)), np.uint8), 64),
}
SHAPES = [(0, 0, -1, -1), (4, 0, 1, -1), (4, 2, 0, 3), (2, 0, -1, -1), (2, 4, 1, 0), (1, 0, -1, -1)]


@pytest.mark.parametrize("name", list(CASES))
def test_matches_oracle(name):
    n, plates, make, P = CASES[name]
    pk = _packed(n, plates, make, seed=7)
    ch = instances.chromosomes(P, n, 11)
    ref, rlog = oracle_decode(pk, ch, n_threads=8, with_log=True)
    torch, dec = _decoder(pk, P)
    chrom = torch.from_numpy(ch).cuda()
    for shape in SHAPES:
        dec.set_launch_config(*shape)
        log = torch.full((P, pk.n_machines, n, 5), -7, dtype=torch.int32, device="cuda")
        for _ in range(2):  # the second launch finds the first one's plates in the workspace
            out = dec.decode(chrom, log=log)
        torch.cuda.synchronize()
        assert int(dec.status.item()) == abi.OK, shape
        np.testing.assert_array_equal(out.cpu().numpy(), ref, err_msg=str(shape))
        got = log.cpu().numpy().reshape(-1).view(abi.PLACEMENT_DTYPE).reshape(rlog.shape)
        assert (got == rlog).all(), shape
