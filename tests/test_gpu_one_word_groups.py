"""The one-word residue kinds in warp groups of 64 terms: range sums bit-exact
against the oracle around m = 2^17 and 2^25 (starts of three and four exponent bits),
2^28, 2^29 (lazy -> middle steps), 2^31 and 2^32, at
group and tile remainders, where a group's exponents cross a multiple of 2^16, at the
end of the main body, and under exponents of 46 bits and more."""
import random

import pytest

pytestmark = pytest.mark.gpu


def check(ctx, oracle, f, d, k0, k1):
    ctx.Set0mem()
    ctx.BatchCalc(k0, k1, f, d)
    want = oracle.sum_range(d, f, k0, k1, 3)
    if k1 == d:
        want += oracle.sum_range(d, f, d, d + 20, 3)
    assert ctx.read_partial() == want % (1 << 192), (f, d, k0, k1)


def first_k(oracle, f, m):
    return (m - oracle.DEN1[f] + oracle.DEN0[f] - 1) // oracle.DEN0[f]


@pytest.mark.parametrize("limit", [17, 25, 28, 29, 31, 32])
@pytest.mark.parametrize("f", [0, 4])
def test_range_sums_at_the_limits(ctx192, oracle, f, limit):
    rng = random.Random(limit)
    k = first_k(oracle, f, 1 << limit)
    for n in (1, 33, 63, 64, 65, 2047, 2049, 5000):
        for d in (k + n + rng.randrange(1, 50), 2 * k + 1, 10 ** 13):
            check(ctx192, oracle, f, d, k - n // 2, k - n // 2 + n)


@pytest.mark.parametrize("limit", [16.5, 24, 27, 28.9, 30, 31.6])
def test_groups_across_a_prefix_boundary(ctx192, oracle, limit):
    for f in (1, 5):
        k = first_k(oracle, f, int(2 ** limit))
        d = k + 123456789
        while (10 * (d - k) + 160) % (1 << 16) > 640:
            k += 1
        for shift in range(0, 64, 9):
            check(ctx192, oracle, f, d, k - shift, k - shift + 3500)


@pytest.mark.parametrize("d", [1, 3, 7, 31, 32, 33, 63, 65, 127, 1639, 1663, 26240, 400001])
def test_short_series_to_the_end(ctx192, oracle, d):
    """Exponents down to 10 in the last groups before d."""
    for f in range(7):
        check(ctx192, oracle, f, d, max(0, d - 700), d)
