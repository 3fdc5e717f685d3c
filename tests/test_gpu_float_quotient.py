"""The float-quotient two-word steps (2^32 <= m < 94 * 2^32): terms and range sums
bit-exact against the oracle at the limits of their ranges, at warp-group and tile
remainders, and where a group's exponents cross a multiple of 2^16."""
import random

import pytest

pytestmark = pytest.mark.gpu

LOW, HIGH = 15 << 34, 94 << 32
E_CROSS = 1 << 16                                        # exponents agree above bit 16 or run singly


def first_k(oracle, f, m):
    return (m - oracle.DEN1[f] + oracle.DEN0[f] - 1) // oracle.DEN0[f]


@pytest.mark.parametrize("limit", [1 << 32, LOW, HIGH])
@pytest.mark.parametrize("f", [0, 2, 6])
def test_terms_at_the_limits(ctx192, oracle, f, limit):
    k = first_k(oracle, f, limit)
    for d in (k + 45, 10 * k + 1):
        ks = list(range(k - 40, k + 40))
        for kk, g in zip(ks, ctx192.terms(d, f, ks)):
            assert g == oracle.term(d, f, kk, 3), (d, f, kk)


@pytest.mark.parametrize("n", [1, 31, 32, 63, 64, 65, 127, 2047, 2048, 2049, 9001])
@pytest.mark.parametrize("limit", [1 << 32, LOW, HIGH])
def test_range_sums_at_the_limits(ctx192, oracle, limit, n):
    rng = random.Random(n + limit)
    for f in (1, 3):
        k = first_k(oracle, f, limit)
        for d in (k + n + rng.randrange(1, 40), 3 * k + 7):
            for k0 in (k, k - n, k - n // 2):
                ctx192.Set0mem()
                ctx192.BatchCalc(k0, k0 + n, f, d)
                assert ctx192.read_partial() == oracle.sum_range(d, f, k0, k0 + n, 3), (f, d, k0, n)


@pytest.mark.parametrize("f", [0, 5])
def test_groups_across_a_prefix_boundary(ctx192, oracle, f):
    """Ranges in which 10 (d - k) + 168 passes a multiple of 2^16 at every offset
    inside a group of 64 terms (one term in 6554 starts a new prefix)."""
    d = 39999999999
    k = first_k(oracle, f, 3 << 33)
    while (10 * (d - k) + 168) % E_CROSS > 640:
        k += 1
    for shift in range(0, 64, 9):
        k0 = k - shift
        ctx192.Set0mem()
        ctx192.BatchCalc(k0, k0 + 7000, f, d)
        assert ctx192.read_partial() == oracle.sum_range(d, f, k0, k0 + 7000, 3)


@pytest.mark.parametrize("d", [4 * 10 ** 13 - 1, 399999999999999997])
def test_long_exponents(ctx192, oracle, d):
    """Small two-word moduli under exponents up to 2^62."""
    for f in (1, 6):
        for m in (1 << 32, 1 << 36, HIGH - 50000):
            k = first_k(oracle, f, m)
            ctx192.Set0mem()
            ctx192.BatchCalc(k, k + 2500, f, d)
            assert ctx192.read_partial() == oracle.sum_range(d, f, k, k + 2500, 3), (f, m)
