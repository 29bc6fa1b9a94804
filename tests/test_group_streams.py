"""The window lists and streams of a template group (csrc/fbp_lik_tcw.cuh, k_tcw_count
and k_tcw_lists), restated thread by thread: a thread takes 16 windows and the two
beside them as bits of a word, a block 4096 windows.  Checked against the plain
definition -- window i of the list stands at i L + (runs before it) (L - 1) -- and for
what the tiles rely on: every tile of the stream has a first window that starts at or
before it, no tile meets more windows than its table holds, and every kept output
lies in exactly one tile."""
import numpy as np
import pytest

WPOS, PER, TILE = 2048, 16, 4096


def staged(L):             # positions of a tile that are staged
    return WPOS + 16 * ((L + 7 + 15) // 16)


def entries(L):            # windows that a tile's table holds
    return min(staged(L) // L + 3, 136)


def thread_bits(sel, base):
    W = len(sel)
    m = int(base > 0 and base - 1 < W and sel[base - 1])
    for k in range(PER + 1):
        m |= int(base + k < W and sel[base + k]) << (k + 1)
    return m


def lists(sel, L):
    W = len(sel)
    blocks = -(-W // TILE)
    bits = [[thread_bits(sel, b * TILE + t * PER) for t in range(TILE // PER)] for b in range(blocks)]
    own = (1 << PER) - 1

    def counts(m):
        mine, prev = (m >> 1) & own, m & own
        return mine.bit_count(), (mine & ~prev).bit_count()
    per_block = [tuple(map(sum, zip(*map(counts, row)))) for row in bits]
    win, pos, first = {}, {}, {}
    for b in range(blocks):
        i0 = sum(c[0] for c in per_block[:b])
        r0 = sum(c[1] for c in per_block[:b])
        for t, m in enumerate(bits[b]):
            i = i0 + sum(counts(x)[0] for x in bits[b][:t]) if m >> 1 & own else 0
            runs = r0 + sum(counts(x)[1] for x in bits[b][:t]) if m >> 1 & own else 0
            for k in range(PER):
                if not m >> (k + 1) & 1:
                    continue
                if not m >> k & 1:
                    runs += 1
                p = i * L + (runs - 1) * (L - 1)
                win[i], pos[i] = b * TILE + t * PER + k, p
                nxt = p + L + (0 if m >> (k + 2) & 1 else L - 1)
                q = (p + WPOS - 1) // WPOS
                if q * WPOS < nxt:
                    assert q not in first
                    first[q] = i
                i += 1
    n, r = (sum(c[k] for c in per_block) for k in (0, 1))
    tiles = ((n - 1) * L + (r - 1) * (L - 1) + L + WPOS - 1) // WPOS if n else 0
    return win, pos, first, n, tiles


@pytest.mark.parametrize("L", [16, 17, 31, 61, 101, 150, 190, 200, 260, 329])
@pytest.mark.parametrize("density", [0.0, 0.02, 0.3, 0.9, 1.0])
def test_lists_and_streams(L, density):
    r = np.random.Generator(np.random.PCG64(L * 10 + int(10 * density)))
    for W in (1, 15, 16, 17, 300, TILE - 1, TILE + 1, 2 * TILE + 40):
        sel = r.random(W) < density
        if density and W > TILE:
            sel[TILE - 2:TILE + 2] = True            # a run over a block's end
        win, pos, first, n, tiles = lists(sel, L)
        w = np.nonzero(sel)[0]
        assert n == len(w) and [win[i] for i in range(n)] == w.tolist()
        if n == 0:
            assert tiles == 0
            continue
        start = np.concatenate([[True], np.diff(w) != 1])
        p = np.arange(n) * L + (np.cumsum(start) - 1) * (L - 1)
        assert [pos[i] for i in range(n)] == p.tolist()
        assert tiles == -(-(p[-1] + L) // WPOS)
        for q in range(tiles):
            i = first[q]
            assert p[i] <= q * WPOS
            # the windows before it end, with the lags of a run's last outputs, before the tile
            assert i == 0 or p[i] <= q * WPOS < (p[i + 1] if i + 1 < n else p[i] + 2 * L - 1)
            assert np.searchsorted(p, q * WPOS + staged(L)) - i <= entries(L)
        kept = (p[:, None] + np.arange(L)).ravel()
        assert len(np.unique(kept)) == n * L and kept.max() < tiles * WPOS
