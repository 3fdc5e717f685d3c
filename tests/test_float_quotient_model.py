"""The float-quotient ladder step in exact arithmetic: for moduli over the whole
range and residues at both ends of theirs, the product stays in one 64-bit word,
divisible by 2^24, and the next residue within the bounds that the step assumes."""
import random
from fractions import Fraction

import pytest


def round_down(x: Fraction) -> Fraction:
    """x > 0 rounded down to a float's 24 significant bits."""
    e = x.numerator.bit_length() - x.denominator.bit_length() - 24
    while x / Fraction(2) ** e >= 1 << 24:
        e += 1
    while x / Fraction(2) ** e < 1 << 23:
        e -= 1
    return Fraction(int(x / Fraction(2) ** e)) * Fraction(2) ** e


def root_below(m: int, ulps: int) -> Fraction:
    """2^6 / sqrt(m) rounded down to 24 bits, less a number of last places."""
    e = 0
    while (1 << 12 << 2 * e) < (1 << 46) * m:                # 24 bits: root in [2^23, 2^24)
        e += 1
    from math import isqrt
    return Fraction(isqrt((1 << 12 << 2 * e) // m) - ulps, 1 << e)


@pytest.mark.parametrize("offset,low,high", [(2, 1 << 32, 15 << 34), (1, 15 << 34, 94 << 32)])
def test_step_bounds(offset, low, high):
    rng = random.Random(high)
    bound = Fraction(0)
    for i in range(600):
        m = (high - 1 - 2 * rng.randrange(50), low + 1 + 2 * rng.randrange(50), rng.randrange(low, high) | 1)[i % 3]
        s = root_below(m, rng.randrange(3))
        zmax = Fraction(395 if offset == 2 else 265, 100)
        for y in (int(2 * zmax * m) - rng.randrange(99), (offset - 1) * m + 1 + rng.randrange(99),
                  rng.randrange((offset - 1) * m + 1, int(2 * zmax * m))):
            assert y < 1 << 41
            t = round_down(s * (y >> 18)) if y >> 18 else Fraction(0)
            q = int(round_down(t * t + (1 << 23)) - (1 << 23)) if t * t >= 1 else 0
            u = y * y * pow(m, -1, 1 << 24) % (1 << 24)
            x = y * y - (u + ((q - offset) << 24)) * m
            assert 0 <= x < 1 << 64 and x % (1 << 24) == 0
            z = x >> 24
            assert (offset - 1) * m <= z < zmax * m
            assert -1 <= q - offset < 1 << 22
            bound = max(bound, Fraction(z, m))
    assert bound > zmax - Fraction(1, 2)                     # the bound is nearly met
