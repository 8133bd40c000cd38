# SPDX-License-Identifier: Apache-2.0
"""The index arithmetic of the cube passes, restated on the CPU and checked against brute force:
cube_ext.cu covers the window of every output with a block suffix H, a block prefix G and two table
entries (or block starts) inside the arrays; cube_box.cu finds the segment, chunk and carry of every
output's G and H by a multiply-high, and every slot and total lies inside the CTA's buffers."""

from __future__ import annotations

import random

import pytest


def mulhi(u: int, inv: int) -> int:
    assert 0 <= u < 2**32
    return (u * inv) >> 32


def block_cap(n: int, P: int, rows: bool) -> int:
    if not rows:
        return 15 if n <= 640 else 31
    return 16 if P == 8 else (20 if n <= 640 else 28)


def block_len(r: int, cap: int, P: int, rows: bool) -> int:
    if 2 * r >= cap:
        return cap
    if rows and P != 8:
        return 4 if r < 6 else 12
    two = 2 << (r.bit_length() - 1)
    return two if rows else two - 1


def table_elems(n: int, P: int, rows: bool) -> int:
    nb = -(-n // block_cap(n, P, rows))
    k = 1
    while (2 << (k - 1)) <= nb - 1:
        k += 1
    return nb * k


def lengths(rng: random.Random):
    return rng.choice([2, 3, 15, 16, 19, 20, 21, 31, 32, 60, 61, 62, 639, 640, 641, rng.randint(2, 100), rng.randint(2, 3000)])


@pytest.mark.parametrize("P,rows", [(8, True), (1, True), (8, False)])
def test_extremes_cover_the_window(P, rows):
    rng = random.Random(7)
    for _ in range(400):
        n = lengths(rng)
        longest = n if rng.random() < 0.5 else n + rng.randint(0, n)  # a batch of uneven lengths: sized for the longest
        r = min(rng.choice([2, 3, 4, 5, 6, 7, 8, 9, 10, 13, 14, 15, 16, rng.randint(2, 64), rng.randint(2, 2 * n)]), n - 1)
        if r < 2:
            continue
        cap = block_cap(longest, P, rows)
        B = block_len(r, cap, P, rows)
        assert B <= 2 * r and (B % 4 == 0 if rows else B % 2 == 1)
        if rows and P == 8:  # a warp step is a whole number of blocks
            assert 32 % B == 0
        inv = 0xFFFFFFFF // B + 1
        nb = -(-n // B)
        levels, most = 1, min(nb - 1, 2 * r // B)
        while B == cap and (2 << (levels - 1)) <= most:
            levels += 1
        assert B < cap or levels * nb <= table_elems(longest, P, rows)
        block_end = lambda i: min(i // B * B + B, n)  # noqa: E731
        for x in range(n):
            lo, hi = x - r, min(x + r, n - 1)
            b0 = mulhi(lo, inv) if lo >= 0 else -1
            b1 = mulhi(hi, inv)
            assert b1 == hi // B and (lo < 0 or b0 == lo // B)
            seen = set()
            if lo >= 0:
                seen |= set(range(lo, block_end(lo)))
            if b1 > b0:
                seen |= set(range(b1 * B, hi + 1))
            L = b1 - b0 - 1
            if L > 0:
                if B == cap:
                    k = L.bit_length() - 1
                    assert k < levels
                    starts, count = (b0 + 1, b1 - (1 << k)), 1 << k
                else:
                    assert L <= 2
                    starts, count = (b0 + 1, b1 - 1), 1
                for s in starts:
                    assert 0 <= s < nb and s + count <= nb
                    seen |= set(range(s * B, min((s + count) * B, n)))
            assert seen == set(range(max(lo, 0), hi + 1)), (n, r, x)


@pytest.mark.parametrize("wide", [False, True])
def test_box_outputs_find_their_segments_and_carries(wide):
    rng = random.Random(11)
    for _ in range(400):
        n = rng.choice([17000, 8191]) if wide and rng.random() < 0.05 else lengths(rng)
        w = 2 * (rng.randint(1, 2 * n) if wide else rng.randint(1, 70)) + 1
        r = min((w - 1) // 2, n - 1)
        wa = 2 * r + 1
        if wa == 1:
            continue
        o = (n * ((wa + 1) // 2)) % wa
        assert o == ((n >> 1) + (n & 1) * (r + 1)) % wa  # its 32-bit form
        k_lo, k_hi = (r - o) // wa, (n - 1 + r - o) // wa
        nseg, cps = k_hi - k_lo + 1, (wa + 31) >> 5
        assert cps == 1 or nseg * cps <= n // 8 + 24  # tot_slots
        inv = 0xFFFFFFFF // wa + 1
        ug = r - o - k_lo * wa
        uh = n - 1 + ug
        first = o + k_lo * wa
        assert first >= -n and n - 1 + r < 2 * n  # one reflection
        for x in range(n) if n < 4000 else random.Random(x0 := n).sample(range(n), 500):
            for u, e in ((x + ug, x + r), (uh - x, n - 1 - x + r)):
                k = mulhi(u, inv)
                m = u - k * wa
                assert 0 <= m < wa and 0 <= k < nseg
                s = o + (k_lo + k) * wa
                assert s + m == e and (m >> 5) < cps
                assert (m == wa - 1) == (e == s + wa - 1)


def test_panel_divisions_are_exact():
    rng = random.Random(3)
    for _ in range(20000):
        d = rng.randint(1, rng.choice([2, 64, 3000, 2**31 - 1]))
        s = 0
        while (1 << s) < d:
            s += 1
        m = ((1 << 32) * ((1 << s) - d) // d + 1) & 0xFFFFFFFF
        for x in (rng.randint(0, 2**31 - 1), rng.randint(0, 2**16), d - 1, d, min(2**31 - 1, 2 * d - 1), 2**31 - 1):
            total = ((x * m) >> 32) + x
            assert total < 2**32 and total >> s == x // d
