# SPDX-License-Identifier: Apache-2.0
"""The index arithmetic of the tiled long-line passes (cube_long.cu), restated on the CPU: a max / min
tile covers every output's window with the block suffixes, prefixes and runs of blocks that it holds;
a box tile finds every output's segment, chunk and carry in the parts of the line that it stages, and
its buffers hold them, for short segments (folded in the tile) and long ones (carries from the table);
the table holds the chunks of every window."""

from __future__ import annotations

import random

import pytest


def lines(rng: random.Random, tile: int):
    n = rng.choice([rng.randint(2, 400), rng.randint(2000, 9000), rng.randint(9000, 65536), 65536, 16384, 20001])
    w = 2 * rng.choice([rng.randint(1, 20), rng.randint(1, 600), rng.randint(1, 65535)]) + 1
    return n, min((w - 1) // 2, n - 1), rng.randrange((n + tile - 1) // tile)


@pytest.mark.parametrize("tile", [1024, 4096])
def test_extreme_tiles_cover_their_windows(tile):
    rng = random.Random(tile)
    for _ in range(500):
        n, r, t = lines(rng, tile)
        if r < 1:
            continue
        X0, X1 = t * tile, min(t * tile + tile, n)
        B = 32 if r >= 16 else 2 << (r.bit_length() - 1)
        assert B <= 2 * r
        sh, nb, span = B.bit_length() - 1, (n + 31) >> 5, tile + 128
        h0 = (max(X0 - r, 0) >> 5) << 5
        h1 = min(n, ((max(X1 - 1 - r, 0) + 2 * B) >> 5) * 32 + 32)
        g0 = (min(X0 + r, n - 1) >> 5) << 5
        g1 = min(n, (min(X1 - 1 + r, n - 1) >> 5) * 32 + 32)
        assert ((h1 - h0 + 31) // 32) * 32 <= span and ((g1 - g0 + 31) // 32) * 32 <= span
        run, least = 0, (r >> 4) - 1
        while B == 32 and (2 << run) <= least:
            run += 1
        end_of = lambda i: min((i // B) * B + B, n)  # noqa: E731
        blocks = lambda j: (j, min(j + (1 << run), nb))  # noqa: E731  blocks of S[j]
        for x in sorted({X0, X0 + 1, X1 - 1, *(rng.randrange(X0, X1) for _ in range(60))} & set(range(X0, X1))):
            lo, hi = x - r, min(x + r, n - 1)
            b0, b1 = (lo >> sh if lo >= 0 else -1), hi >> sh
            parts = []
            if lo >= 0:
                assert h0 <= lo < h1
                parts.append((lo, end_of(lo)))
            if b1 > b0:
                assert g0 <= hi < g1
                parts.append((b1 * B, hi + 1))
            if b1 - b0 > 1:
                if B < 32:
                    s = (b0 + 1) << sh
                    assert b1 - b0 == 2 and h0 <= s < h1
                    parts.append((s, end_of(s)))
                elif lo < 0:
                    assert X0 < r and b1 - 1 < nb
                    parts.append((0, b1 * 32))
                else:
                    for j in (b0 + 1, max(b0 + 1, b1 - (1 << run))):
                        assert 0 <= j < nb
                        u, v = blocks(j)
                        parts.append((u * 32, min(v * 32, n)))
            parts.sort()
            at = max(lo, 0)
            assert parts[0][0] == at and max(v for _, v in parts) == hi + 1, (n, r, x)
            for u, v in parts:
                assert at <= u <= at or u <= at, (n, r, x, parts)
                at = max(at, v)


def side(wa, cps, first, p0, p1, wide):
    k0 = (p0 - first) // wa
    in0 = p0 - first - k0 * wa
    skip = in0 >> 5 if wide else 0
    e0 = first + k0 * wa + 32 * skip
    k1 = (p1 - first) // wa
    chunks = (k1 - k0) * cps + ((p1 - first - k1 * wa) >> 5) - skip + 1
    return k0, skip, e0, p1 - e0 + 1, chunks


@pytest.mark.parametrize("tile", [1024, 4096])
def test_box_tiles_hold_their_segments(tile):
    rng = random.Random(tile + 1)
    samples = tile + tile // 4 + 32
    most_chunks = samples // 2 + 8
    for _ in range(700):
        n, r, t = lines(rng, tile)
        wa = 2 * r + 1
        if wa == 1:
            continue
        X0, X1 = t * tile, min(t * tile + tile, n)
        o = ((n >> 1) + (n & 1) * (r + 1)) % wa
        k_lo, k_hi = (r - o) // wa, (n - 1 + r - o) // wa
        nseg, cps = k_hi - k_lo + 1, (wa + 31) >> 5
        first, e_max = o + k_lo * wa, n - 1 + r
        wide = wa > tile // 4
        assert not wide or nseg * cps <= n // 8 + 24  # the table of chunk totals
        for p0, p1 in ((X0 + r, X1 - 1 + r), (n - X1 + r, n - 1 - X0 + r)):
            assert p0 >= first and p1 <= e_max and first >= -n
            k0, skip, e0, length, chunks = side(wa, cps, first, p0, p1, wide)
            assert length <= samples and chunks <= most_chunks and e0 <= p0
            inv = 0xFFFFFFFF // wa + 1
            held = {}
            for q in range(chunks):  # the fold tasks: chunk -> its samples
                k, c = divmod(q + skip, cps)
                s0 = first + (k0 + k) * wa
                c0 = s0 + 32 * c
                c1 = min(c0 + 31, s0 + wa - 1, e_max, e0 + length - 1)
                held[(k, c)] = (c0, c1)
            for e in {p0, p1, *(rng.randint(p0, p1) for _ in range(20))}:
                m = e - (first + k0 * wa)
                k = m // wa if wide else (m * inv) >> 32
                assert k == m // wa
                m -= k * wa
                c0, c1 = held[(k, m >> 5)]
                assert c0 <= e <= c1 and c0 == first + (k0 + k) * wa + 32 * (m >> 5)
                if wide:
                    assert (k0 + k) * cps + (m >> 5) < nseg * cps
                else:  # every earlier chunk of the segment is folded whole
                    for c in range(m >> 5):
                        a, b = held[(k, c)]
                        assert (a, b) == (first + (k0 + k) * wa + 32 * c, a + 31)


def test_windows_of_several_chunks_fit_the_table_of_totals():
    """The chunk totals of a window's segments (nseg cps, when a segment has more than one chunk) fit the
    tot_slots(n) = n / 8 + 24 that the box passes and the long lines' carries hold per line and direction."""
    rng = random.Random(11)
    for _ in range(200000):
        n = rng.randint(2, 65536)
        r = min(rng.randint(0, rng.choice([20, 200, 5000, 70000])), n - 1)
        wa, cps = 2 * r + 1, (2 * r + 1 + 31) >> 5
        o = ((n >> 1) + (n & 1) * (r + 1)) % wa
        nseg = (n - 1 + r - o) // wa - (r - o) // wa + 1
        assert cps == 1 or nseg * cps <= n // 8 + 24, (n, r, nseg, cps)
