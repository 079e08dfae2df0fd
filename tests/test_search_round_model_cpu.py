"""CPU model of one chunk of the decode kernel's plate search (search_plate in
brkga_fft2_b200/csrc/brkga_decoder.cu), lane by lane: how the pairs of a
surviving row and 64 candidate columns are dealt to the lanes, the pieces that
groups of lanes test, the whole warp's test of the pairs left open, and the key
that decides.  Checked against trying every row and column in the order of the
keys, for every number of open pairs and pieces, with the coarse test passing
anything between all pairs and none that is blocked."""
import numpy as np
import pytest

LANES, GROUP_OPEN, GROUP_SEGS = 32, 3, 4
MAX_SIDE = 8191
M64 = (1 << 64) - 1


def row_key(newlen, y):
    return newlen << 13 | (MAX_SIDE - y)


def key_of(row, x, r):
    return row << 32 | x << 2 | r


def dealt(ntask, nw):
    """(survivor, word) of the pairs in the order the lanes take them."""
    inv = 0xFFFFFFFF // nw + 1 if nw > 1 else 0
    out = []
    for t in range(ntask):
        si = (t * inv) >> 32 if nw > 1 else t
        out.append((si, t - si * nw))
    return out


@pytest.mark.parametrize("nw", list(range(1, 12)) + [16, 31, 32, 63, 64, 100, 127, 128])
def test_pairs_are_dealt_row_after_row(nw):
    ntask = 32 * nw
    assert dealt(ntask, nw) == [(t // nw, t % nw) for t in range(ntask)]


def chunk(pairs, pieces, gseg, best):
    """The kernel's rounds over `pairs`: (key bound, open columns after the coarse test, blocked columns per piece)
    each; `best`: the key to beat.  Returns the best key, the way search_plate leaves it."""
    for t0 in range(0, len(pairs), LANES):
        rnd = pairs[t0:t0 + LANES]
        if rnd[0][0] >= best:
            break
        F = [p[1] for p in rnd] + [0] * (LANES - len(rnd))
        opened = sum(1 << i for i in range(LANES) if F[i])
        n_open, q0 = bin(opened).count("1"), 0
        if n_open >= GROUP_OPEN and gseg:
            lg = 3 if n_open <= 4 else 2 if n_open <= 8 else 1 if n_open <= 16 else 0
            n = min(max(gseg, 1 << lg), pieces)
            left = [None] * LANES
            srcs = []
            for lane in range(LANES):
                m = opened
                if lg:
                    for k in range((32 >> lg) - 1):
                        if k < lane >> lg:
                            m &= m - 1 if m else 0
                else:
                    m &= 1 << lane
                src = (m & -m).bit_length() - 1 if m else 0
                srcs.append((src, bool(m)))
                f = F[src] if m else 0
                q = lane & ((1 << lg) - 1)
                while q < n and f:
                    f &= ~rnd[src][2][q] if src < len(rnd) else 0
                    q += 1 << lg
                left[lane] = f & M64
            for o in (1, 2, 4):  # the exchanges inside a group
                if o < 1 << lg:
                    left = [left[i] & left[i ^ o] for i in range(LANES)]
            new = []
            for lane in range(LANES):
                frm = bin(opened & ((1 << lane) - 1)).count("1") << lg if lg else lane
                if opened >> lane & 1:  # the value comes from this pair's own group
                    assert srcs[frm & 31] == (lane, True)
                new.append(F[lane] & left[frm & 31])
            F = new
            opened &= sum(1 << i for i in range(LANES) if F[i])
            q0 = max(gseg, 1 << lg)
        while opened:
            l = (opened & -opened).bit_length() - 1
            opened &= opened - 1
            if rnd[l][0] >= best:
                break
            f = F[l]
            for q in range(q0, pieces, 32):
                if not f:
                    break
                blocked = 0
                for lane in range(LANES):
                    if q + lane < pieces:
                        blocked |= rnd[l][2][q + lane]
                f &= ~blocked & M64
            if f:
                return min(best, rnd[l][0] + (((f & -f).bit_length() - 1) << 2))
    return best


def direct(pairs, best):
    keys = []
    for bound, f, blocked in pairs:
        for b in blocked:
            f &= ~b & M64
        if f:
            keys.append(bound + (((f & -f).bit_length() - 1) << 2))
    return min(keys + [best])


@pytest.mark.parametrize("gseg", [0, 4, 7, 20])
@pytest.mark.parametrize("dens", [0.005, 0.03, 0.12, 0.5])
def test_chunk_finds_the_smallest_key(gseg, dens):
    rng = np.random.default_rng([gseg, int(1000 * dens)])
    for trial in range(150):
        pieces = int(rng.choice([1, 2, 3, 4, 5, 8, 9, 31, 32, 33, 36, 70, 140]))
        nw, rows = int(rng.integers(1, 5)), int(rng.integers(1, 33))
        L, h, r, enc = 200, int(rng.integers(1, 60)), int(rng.integers(0, 4)), int(rng.integers(0, 200))
        ty_hi = L - h
        surv = sorted(rng.choice(32, size=rows, replace=False).tolist())
        pairs = []
        for si, k in dealt(rows * nw, nw):
            ty = ty_hi - surv[si]
            if ty < 0:
                continue
            bits = rng.random((pieces, 64)) < dens * rng.choice([0.2, 1.0, 3.0])
            blocked = [int(np.packbits(b[::-1]).view(">u8")[0]) for b in bits]
            free = M64
            for b in blocked:
                free &= ~b & M64
            # the coarse test may leave any blocked column open, never close a free one
            f = free | int(rng.integers(0, 1 << 63)) * 2 if rng.random() < 0.7 else free
            if rng.random() < 0.2:  # the last word of a row: fewer columns
                f &= (1 << int(rng.integers(1, 64))) - 1
            pairs.append((key_of(row_key(max(enc, L - ty), ty + h - 1), 64 * k, r), f, blocked))
        if not pairs:
            continue
        bounds = [p[0] for p in pairs]
        assert bounds == sorted(bounds)  # pairs come in the order of their keys
        assert all(a + (63 << 2) < b for a, b in zip(bounds, bounds[1:]))  # and no pair reaches into the next one's
        none = (1 << 64) - 1
        for best in (none, bounds[len(bounds) // 2], bounds[-1] + 1):
            assert chunk(pairs, pieces, gseg, best) == direct(pairs, best)


def test_rows_compare_as_the_keys_upper_word():
    """Smaller newLen first, then the larger bottom row, the smaller column, the first rotation."""
    rng = np.random.default_rng(3)
    pts = [(int(rng.integers(1, 8192)), int(rng.integers(0, 8191)), int(rng.integers(0, 8191)), int(rng.integers(0, 4)))
           for _ in range(400)]
    by_key = sorted(pts, key=lambda p: key_of(row_key(p[0], p[1]), p[2], p[3]))
    assert by_key == sorted(pts, key=lambda p: (p[0], -p[1], p[2], p[3]))
    assert key_of(row_key(8191, 0), 8191, 3) < 1 << 64
