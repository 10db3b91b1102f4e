"""The stratified decision from the reciprocal's fraction bits, restated in
exact integers: wherever the bits are taken to decide, they decide as the
exact test does (words next to the boundary included)."""
import random

import pytest

M32 = (1 << 32) - 1


def _product(C, m):
    """B of pf32_dev.cuh: the high half of C m from three 32 x 32 products."""
    c1, c0, m1, m0 = C >> 32, C & M32, m >> 32, m & M32
    return c1 * m1 + ((c1 * m0) >> 32) + ((c0 * m1) >> 32)


@pytest.mark.parametrize("n", [2, 31, 1000, 16384, 100003, (1 << 24) + 7,
                               (1 << 30) - 1])
def test_fraction_bits_decide_as_the_exact_test(n):
    rng = random.Random(n)
    decided = asked = 0
    for _ in range(3000):
        # totals of the filters: the largest weight alone is 2^K
        K = 63 - max(1, (n - 1).bit_length())
        Q = rng.randint(1 << K, min(n << K, (1 << 63) - 1))
        s = 32
        while s > 0 and (n << s) >= Q:
            s -= 1
        assert s >= 20
        m = ((n << s) << 64) // Q
        C = rng.randint(0, Q - 1)
        if rng.random() < 0.3:  # next to a uniform's cell boundary
            C = min(Q - 1, max(0, rng.randint(0, n) * Q // n
                               + rng.randint(-2, 2)))
        B = _product(C, m)
        mask = (1 << s) - 1
        bl = B & M32
        if ((bl + 6) & mask) < 8:
            continue  # settled exactly
        j, frac = B >> s, bl & mask
        assert j == C * n // Q
        asked += 1
        edge = (frac << (32 - s)) & M32
        words = [0, M32, rng.randint(0, M32)]
        words += [(edge + (d << (32 - s)) + rng.randint(0, (1 << (32 - s)) - 1))
                  & M32 for d in range(-8, 9)]
        for a in words:
            exact = -(-(a * Q) // (1 << 32)) <= C * n - j * Q
            top = a >> (32 - s)
            if ((frac - top + 4) & M32) <= 5:
                continue  # settled exactly
            decided += 1
            assert (top <= ((frac - 2) & M32)) == exact, (Q, C, a)
    assert asked > 1000 and decided > 10 * asked
