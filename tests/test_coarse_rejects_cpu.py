"""The coarse test's tables reject blocked positions: solid masks have cores at
both block heights and at every offset from two blocks of rows on, and on plates
that hold parts most blocked positions fail the test.  The model is the one that
is checked against the direct collision test in test_coarse_test_model_cpu.py;
that test asks only that no free position is rejected, which a test that rejects
nothing would pass too."""
import numpy as np
import pytest

from brkga_fft2_b200.instances import random_part_mask
from tests.test_coarse_test_model_cpu import PLANES, cores, entries, free_positions, longest_run


@pytest.mark.parametrize("rows", [4, 8])
def test_solid_masks_have_cores_at_every_offset(rows):
    rng = np.random.default_rng(rows)
    for _ in range(20):
        h, w = int(rng.integers(2 * rows - 1, 60)), int(rng.integers(PLANES[0], 90))
        mask = np.ones((h, w), np.uint8)
        for off in range(rows):
            cs = cores(mask, off, rows)
            assert cs and all(c[1:] == (0, w) for c in cs)
            assert len(cs) == (off + h) // rows - (1 if off else 0)


@pytest.mark.parametrize("rows", [4, 8])
@pytest.mark.parametrize("seed", range(3))
def test_most_blocked_positions_are_rejected(rows, seed):
    rng = np.random.default_rng([rows, seed, 9])
    L, W = 70, 97
    plate = np.zeros((L, W), np.uint8)
    for _ in range(5):  # parts at their lowest free position, left to right
        m = random_part_mask(rng, 18, 34)
        ys, xs = np.nonzero(free_positions(plate, m))
        if ys.size:
            k = np.lexsort((xs, -ys))[0]
            plate[ys[k]:ys[k] + m.shape[0], xs[k]:xs[k] + m.shape[1]] |= m
    nb = L // rows  # whole blocks
    block_free = np.array([~plate[b * rows:(b + 1) * rows].any(0) for b in range(nb)])
    vac = [np.subtract(*longest_run(r)[::-1]) for r in block_free]
    blocked = rejected = 0
    for _ in range(3):
        m = random_part_mask(rng, 18, 34)
        h, w = m.shape
        free = free_positions(plate, m)
        for y in range(L - h + 1):
            cs = cores(m, y % rows, rows)
            assert all(y // rows + b < nb for b, _, _ in cs)  # a core's block is whole, the plate's last one too
            passed = np.full(W - w + 1, all(vac[y // rows + b] >= n for b, _, n in cs))
            for c in cs:
                for b, lo, second, p in entries(c):
                    run = np.array([block_free[y // rows + b][x:x + PLANES[p]].all() for x in range(W - PLANES[p] + 1)])
                    x = np.arange(W - w + 1)
                    passed &= run[x + lo] & run[x + lo + second]
            assert not (free[y] & ~passed).any()
            blocked += int((~free[y]).sum())
            rejected += int((~free[y] & ~passed).sum())
    assert blocked > 200
    assert rejected > 0.6 * blocked, (rejected, blocked)
