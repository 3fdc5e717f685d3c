"""The short, general and wide two-word kinds, two ladders a lane: terms and range sums
bit-exact against the oracle at m = 39 * 2^40 (18-bit second step -> general step), 2^44 and
2^60, at group and tile remainders, across a multiple of 2^16 in a group's exponents, and
under exponents below and above 2^48."""
import random

import pytest

pytestmark = pytest.mark.gpu

LIMITS = [94 << 32, 1 << 44, 39 << 40, 1 << 60]


def first_k(oracle, f, m):
    return (m - oracle.DEN1[f] + oracle.DEN0[f] - 1) // oracle.DEN0[f]


def check(ctx, oracle, f, d, k0, k1):
    ctx.Set0mem()
    ctx.BatchCalc(k0, k1, f, d)
    assert ctx.read_partial() == oracle.sum_range(d, f, k0, k1, 3), (f, d, k0, k1)


@pytest.mark.parametrize("limit", LIMITS)
@pytest.mark.parametrize("f", [0, 2, 6])
def test_terms_at_the_limits(ctx192, oracle, f, limit):
    k = first_k(oracle, f, limit)
    for d in (k + 45, min(3 * k, 399999999999999997)):
        ks = [x for x in range(k - 40, k + 40) if x < d + 20]
        for kk, g in zip(ks, ctx192.terms(d, f, ks)):
            assert g == oracle.term(d, f, kk, 3), (d, f, kk)


@pytest.mark.parametrize("n", [1, 33, 64, 65, 127, 2049, 6000])
@pytest.mark.parametrize("limit", LIMITS)
def test_range_sums_at_the_limits(ctx192, oracle, limit, n):
    rng = random.Random(n + limit)
    for f in (1, 5):
        k = first_k(oracle, f, limit)
        for d in (k + n + rng.randrange(1, 40), k + 30000000 + rng.randrange(99), min(2 * k, 399999999999999997)):
            for k0 in (k, k - n, k - n // 2):
                check(ctx192, oracle, f, d, k0, k0 + n)


@pytest.mark.parametrize("limit", [(94 << 32) + 1, (39 << 40) - (1 << 20), (39 << 40) + 1])
def test_groups_across_a_prefix_boundary(ctx192, oracle, limit):
    for f in (0, 4):
        k = first_k(oracle, f, limit)
        d = k + 777777777
        while (10 * (d - k) + 142) % (1 << 16) > 640:
            k += 1
        for shift in range(0, 64, 9):
            check(ctx192, oracle, f, d, k - shift, k - shift + 3000)
