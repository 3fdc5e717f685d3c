"""How exact the 106-bit mode's partials are.

Small partials (the tail, the last terms before d) keep a double-double's bits of their own:
their fractions are cut below 2^-192 and summed exactly, and the conversion adds three
double-doubles of one sign, within 2^-103 of the value.

Ranges of ordinary terms: each fraction is cut below 2^-128, sums are exact, and the value,
below 1/2, has its low word (below 2^-54) rounded in five additions, within 2^-104."""
import random
from fractions import Fraction

import pytest

pytestmark = pytest.mark.gpu


def centred(x):
    x %= 1
    return x - 1 if x >= Fraction(1, 2) else x


def partial(ctx):
    hi, lo = ctx.read_partial()
    return centred(Fraction(hi) + Fraction(lo))


@pytest.mark.parametrize("needD", [1000, 10 ** 6, 10 ** 11, 10 ** 16, 999999999999999999])
def test_small_partials_keep_their_bits(ctxdd, oracle, needD):
    d, _ = oracle.pos_to_d(needD)
    for f in range(7):
        den0, den1, sign = oracle.DEN0[f], oracle.DEN1[f], oracle.SIGN[f]
        tail = Fraction(oracle.sum_range(d, f, d, d + 10, 4), 2 ** 256)
        ctxdd.Set0mem()
        ctxdd.Sglobal_after(d, sign, den0, den1)
        ctxdd.Ssum()
        want = centred(tail)
        assert abs(partial(ctxdd) - want) <= abs(want) / 2 ** 103, (f, "tail")
        for before in (1, 2, 3, 6):
            if 1 << (10 * before + 2) > den0 * d:                  # no longer a small sum
                continue
            main = Fraction(oracle.sum_range(d, f, d - before, d, 4), 2 ** 256)
            ctxdd.Set0mem()
            ctxdd.Sglobal64mtg(d - before, d, d, sign, den0, den1)
            ctxdd.Ssum()
            want = centred(main)
            assert abs(partial(ctxdd) - want) <= abs(want) / 2 ** 103, (f, before)
            ctxdd.Set0mem()
            ctxdd.BatchCalc(d - before, d + 20, f, d)
            want = centred(main + tail)
            assert abs(partial(ctxdd) - want) <= abs(want) / 2 ** 103, (f, before, "and tail")


@pytest.mark.parametrize("limit", [1 << 25, 1 << 28, 1 << 31, 1 << 32, 15 << 34, 94 << 32, 1 << 44, 1 << 53, 1 << 60])
def test_ranges_keep_a_double_double(ctxdd, oracle, limit):
    rng = random.Random(limit + 1)
    for f in (1, 3, 6):
        k = (limit - oracle.DEN1[f]) // oracle.DEN0[f]
        for n, gap in ((2, 7), (63, 1), (64, 0), (130, 3), (5000, 6), (40000, 2000)):
            k0 = k - rng.randrange(n + 1)
            d = k0 + n + gap
            ctxdd.Set0mem()
            ctxdd.BatchCalc(k0, k0 + n, f, d)
            want = Fraction(oracle.sum_range(d, f, k0, k0 + n, 4), 2 ** 256)
            if gap == 0:
                want += Fraction(oracle.sum_range(d, f, d, d + 10, 4), 2 ** 256)
            assert abs(centred(partial(ctxdd) - want)) <= Fraction(n, 2 ** 128) + Fraction(1, 2 ** 104), (f, n, gap)


def test_ends_of_short_series(ctxdd, oracle):
    """Series shorter than the terms that are taken with the tail, and split inside them."""
    for d in (1, 3, 5, 7, 9, 15):
        for f in range(7):
            exact = Fraction(oracle.sum_range(d, f, 0, d + 10, 4), 2 ** 256)
            for cut in range(d + 1):
                ctxdd.Set0mem()
                if cut:
                    ctxdd.Sglobal32mtg(0, d, cut, oracle.SIGN[f], oracle.DEN0[f], oracle.DEN1[f])
                ctxdd.BatchCalc(cut, d, f, d)
                assert abs(centred(partial(ctxdd) - exact)) <= Fraction(1, 2 ** 104), (d, f, cut)
