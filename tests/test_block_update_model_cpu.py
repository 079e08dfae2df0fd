"""CPU model of the decode kernel's block update (update_blocks in
brkga_fft2_b200/csrc/brkga_decoder.cu), lane by lane: the group sizes, the steps
of a row wider than 1024 columns and their overlap, the erosions by shuffles,
and the longest run from ballots, on such a row (max_free_run) with the run
carried between steps.  Checked against the planes and the run taken directly
from the block's columns."""
import numpy as np
import pytest

FULL = 0xFFFFFFFF
PLANE_MIN, PLANE_MAX = 2, 5
REACH = (1 << PLANE_MAX) // 32 + 1


def ffs(x):
    return (x & -x).bit_length()


def clz(x):
    return 32 - x.bit_length()


def longest_ones(x):
    return max(len(r) for r in bin(x)[2:].split("0"))


def model(words, n_planes):
    """(planes [n_planes][NW], longest run) of one block, `words` its free columns as 32-bit words."""
    NW = len(words)
    G = 8 if NW <= 8 else 16 if NW <= 16 else 32
    step = 32 if NW <= 32 else 32 - REACH
    planes = [[None] * NW for _ in range(n_planes)]
    best = 0
    for w0 in range(0, NW, step):
        e0 = [words[w0 + g] if w0 + g < NW else 0 for g in range(G)]
        put = [w0 + g < NW and g < step for g in range(G)]
        e = list(e0)
        for k in range(1, PLANE_MAX + 1):
            if k >= PLANE_MIN + n_planes:
                break
            nx = [e[g + 1] if g + 1 < G else 0 for g in range(G)]
            e = [a & (((b << 32 | a) >> (1 << (k - 1))) & FULL) for a, b in zip(e, nx)]
            if k >= PLANE_MIN:
                for g in range(G):
                    if put[g]:
                        planes[k - PLANE_MIN][w0 + g] = e[g]
        if NW > 32:
            continue
        fm = sum(1 << g for g in range(G) if e0[g] == FULL)
        low = [32 if x == FULL else ffs(~x & FULL) - 1 for x in e0]
        for g in range(G):
            rest = ~(fm >> g >> 1) & FULL
            hop = min(ffs(rest) - 1, G - 1 - g)
            end = 0 if g + 1 + hop >= G else low[min(g + 1 + hop, G - 1)]
            best = max(best, longest_ones(e0[g]))
            if e0[g] != FULL or g == 0:
                best = max(best, (32 if e0[g] == FULL else clz(~e0[g] & FULL)) + 32 * hop + end)
    return planes, best if NW <= 32 else max_free_run(words)


def max_free_run(words):
    best, carry = 0, 0
    for w0 in range(0, len(words), 32):
        e = [words[w0 + i] if w0 + i < len(words) else 0 for i in range(32)]
        full = sum(1 << i for i in range(32) if e[i] == FULL)
        low = [32 if x == FULL else ffs(~x & FULL) - 1 for x in e]
        high = [32 if x == FULL else clz(~x & FULL) for x in e]
        before = []
        for i in range(32):
            below = ~full & ((1 << i) - 1)
            at = 31 - clz(below) if below else 0
            before.append(high[at] + 32 * (i - 1 - at) if below else carry + 32 * i)
            best = max(best, longest_ones(e[i]), before[i] + low[i])
        carry = before[31] + 32 if e[31] == FULL else high[31]
    return best


def to_words(cols):
    pad = np.zeros(-(-len(cols) // 32) * 32, np.uint8)
    pad[:len(cols)] = cols
    return [int(x) for x in np.packbits(pad.reshape(-1, 32)[:, ::-1], axis=1).view(">u4").ravel()]


def blocks(W, rng):
    yield np.ones(W, bool)
    yield np.zeros(W, bool)
    for _ in range(30):
        cols = np.ones(W, bool)
        for _ in range(int(rng.integers(1, 6))):  # occupied stretches, at word and step edges too
            x = int(rng.choice([rng.integers(0, W), 32 * rng.integers(0, -(-W // 32)), min(W - 1, 960 * rng.integers(0, 9))]))
            cols[x:x + int(rng.choice([1, 3, 32, 64, 500]))] = False
        yield cols
    yield rng.random(W) < 0.9
    yield rng.random(W) < 0.3


@pytest.mark.parametrize("n_planes", [1, 4])
@pytest.mark.parametrize("W", [1, 31, 32, 33, 250, 256, 257, 512, 513, 1000, 1024, 1025, 1056, 1920, 1921, 1984, 2048, 4000, 8191])
def test_planes_and_longest_run(W, n_planes):
    rng = np.random.default_rng([W, n_planes])
    for cols in blocks(W, rng):
        planes, run = model(to_words(cols), n_planes)
        edges = np.flatnonzero(np.diff(np.concatenate([[0], cols.astype(np.int8), [0]])))
        assert run == (max(edges[1::2] - edges[::2]) if edges.size else 0)
        filled = np.concatenate([[0], np.cumsum(cols)])
        for p in range(n_planes):
            d = 1 << (PLANE_MIN + p)
            at = np.zeros(W, bool)
            if W >= d:
                at[:W - d + 1] = filled[d:] - filled[:-d] == d
            assert planes[p] == to_words(at)
