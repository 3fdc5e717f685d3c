"""The double-double mode's 128-bit fractions: one-series range sums against the exact
256-bit oracle across every residue-kind boundary, odd and even starts, group and tile
remainders. Tolerance 2^-98: at most 312 blocks, so two block partials a thread and eight
tree levels in Ssum, each double-double addition within 2^-104, and truncations below
2^-128 a term."""
import random
from fractions import Fraction

import pytest

pytestmark = pytest.mark.gpu
TOL = Fraction(1, 2 ** 98)


def check(ctx, oracle, f, d, k0, k1):
    ctx.Set0mem()
    ctx.BatchCalc(k0, k1, f, d)
    hi, lo = ctx.read_partial()
    t = (Fraction(hi) + Fraction(lo) - Fraction(oracle.sum_range(d, f, k0, k1, 4), 2 ** 256)) % 1
    assert min(t, 1 - t) < TOL, (f, d, k0, k1, float(min(t, 1 - t)))


@pytest.mark.parametrize("limit", [1 << 25, 1 << 28, 1 << 31, 1 << 32, 15 << 34, 94 << 32, 1 << 44, 1 << 53, 1 << 60])
def test_ranges_across_kind_limits(ctxdd, oracle, limit):
    rng = random.Random(limit)
    for f in (0, 2, 5):
        k = (limit - oracle.DEN1[f]) // oracle.DEN0[f]
        for n in (1, 31, 64, 65, 129, 2500, 20000):
            k0 = k - rng.randrange(n + 1)
            check(ctxdd, oracle, f, k0 + n + 1 + rng.randrange(5000), k0, k0 + n)


def test_short_series(ctxdd, oracle):
    for d in (1, 3, 5, 63, 65, 1001):
        for f in range(7):
            if d > 1:
                check(ctxdd, oracle, f, d, 0, d - 1)


def test_sums_accumulate_over_calls(ctxdd, oracle):
    """Several ranges into one bigSum, of different numbers of blocks."""
    d, f = 3999999999, 3
    ctxdd.Set0mem()
    want = Fraction(0)
    for k0, n in ((5, 1), (430000000, 20000), (429496700, 100), (1000, 7001)):
        ctxdd.Sglobal64mtg(k0, d, k0 + n, oracle.SIGN[f], oracle.DEN0[f], oracle.DEN1[f])
        want += Fraction(oracle.sum_range(d, f, k0, k0 + n, 4), 2 ** 256)
    ctxdd.Ssum()
    hi, lo = ctxdd.read_partial()
    t = (Fraction(hi) + Fraction(lo) - want) % 1
    assert min(t, 1 - t) < TOL


def test_sums_start_from_zero(ctxdd, oracle):
    """Set0mem empties bigSum, whatever an earlier range left in more of its entries."""
    d, f = 3999999999, 2
    ctxdd.Set0mem()
    ctxdd.BatchCalc(1000, 3000000, f, d)
    ctxdd.Set0mem()
    ctxdd.Ssum()
    assert ctxdd.read_partial() == (0.0, 0.0)
    check(ctxdd, oracle, f, d, 500, 620)
    check(ctxdd, oracle, f, d, 500, 20500)
