"""CPU model of the decode kernel's coarse test (coarse_tables, coarse_ok,
coarse_and and update_blocks in brkga_fft2_b200/csrc/brkga_decoder.cu) against
the direct collision test on random plates and masks: at every top row and
column the coarse test may pass a blocked position but must never reject a free
one, whatever the offset of the row in its block, the block height, the plate's
remainders and the mask's shape."""
import numpy as np
import pytest

PLANES = (4, 8, 16, 32)  # runs of the erosion planes


def longest_run(row):
    best, at, j = 0, 0, 0
    while j < len(row):
        if row[j]:
            s = j
            while j < len(row) and row[j]:
                j += 1
            if j - s > best:
                best, at = j - s, s
        else:
            j += 1
    return at, at + best


def cores(mask, off, rows):
    """(block, first column, length) of the blocks a mask covers whole, its top row at offset `off` of a block."""
    h, w = mask.shape
    runs = [longest_run(r) for r in mask]
    out = []
    for i in range((rows - off) % rows, h - rows + 1, rows):
        lo = max(runs[i + k][0] for k in range(rows))
        hi = min(runs[i + k][1] for k in range(rows))
        if hi - lo >= PLANES[0]:
            out.append(((i + off) // rows, lo, hi - lo))
    return out


def entries(core):
    """(block, first column, second window's offset, plane) reads of one core."""
    block, lo, length = core
    at, out = 0, []
    while at < length:
        n = min(length - at, 2 * PLANES[-1])
        if n < PLANES[0]:
            at, n = length - PLANES[0], PLANES[0]
        p = max(k for k, v in enumerate(PLANES) if v <= n)
        out.append((block, lo + at, n - PLANES[p], p))
        at += n
    return out


def free_positions(plate, mask):
    L, W = plate.shape
    h, w = mask.shape
    out = np.zeros((L - h + 1, W - w + 1), bool)
    for y in range(L - h + 1):
        for x in range(W - w + 1):
            out[y, x] = not (plate[y:y + h, x:x + w] & mask).any()
    return out


@pytest.mark.parametrize("rows", [4, 8])
@pytest.mark.parametrize("seed", range(6))
def test_coarse_test_passes_every_free_position(rows, seed):
    rng = np.random.default_rng([rows, seed])
    L, W = int(rng.integers(5, 60)), int(rng.choice([31, 32, 33, 64, 75, 97]))
    plate = np.zeros((L, W), np.uint8)
    for _ in range(int(rng.integers(0, 9))):  # blobs, the lower rows fuller, and single cells
        y, x = int(rng.integers(0, L)), int(rng.integers(0, W))
        plate[y:y + int(rng.integers(1, 14)), x:x + int(rng.integers(1, 24))] = 1
    plate |= (rng.random((L, W)) < rng.choice([0.0, 0.004, 0.02])).astype(np.uint8)
    nb = -(-L // rows)
    block_free = np.array([~plate[b * rows:(b + 1) * rows].any(0) for b in range(nb)])
    vac = [np.subtract(*longest_run(r)[::-1]) for r in block_free]
    planes = np.zeros((len(PLANES), nb, W + 2 * PLANES[-1]), bool)
    for k, n in enumerate(PLANES):
        for x in range(W - n + 1):
            planes[k, :, x] = block_free[:, x:x + n].all(1)
    rejected = tested = 0
    for _ in range(6):
        h, w = int(rng.integers(1, min(L, 40) + 1)), int(rng.integers(1, min(W, 90) + 1))
        mask = (np.abs(np.linspace(-1, 1, w))[None, :] <= rng.uniform(0.3, 1.0, (h, 1))).astype(np.uint8)
        mask[rng.random(h) < 0.05] = 0
        mask[0, 0] = mask[-1, -1] = 1
        free = free_positions(plate, mask)
        for y in range(L - h + 1):
            cs = cores(mask, y % rows, rows)
            passed = np.full(W - w + 1, all(vac[y // rows + b] >= n for b, _, n in cs))
            for c in cs:
                covered = np.zeros(w + 1, bool)
                for b, lo, second, p in entries(c):
                    covered[lo:lo + PLANES[p]] = covered[lo + second:lo + second + PLANES[p]] = True
                    row = planes[p, y // rows + b]
                    x = np.arange(W - w + 1)
                    passed &= row[x + lo] & row[x + lo + second]
                assert covered[c[1]:c[1] + c[2]].all() and covered.sum() == c[2]  # the reads are the core, no more
            assert not (free[y] & ~passed).any()
            tested += passed.size
            rejected += int((~passed).sum())
    assert tested
