"""Two-word groups whose exponents are 2^48 and more, where the bits that a group has in
common take two words: range sums bit-exact against the oracle on both sides of 2^48, at
the longest exponents, and across multiples of 2^16, for each two-word kind."""
import pytest

pytestmark = pytest.mark.gpu

D_MAX = 399999999999999997
KINDS = [(94 << 32) + 1, 1 << 43, (39 << 40) + 1, 1 << 50]


def check(ctx, oracle, f, d, k0, k1):
    ctx.Set0mem()
    ctx.BatchCalc(k0, k1, f, d)
    assert ctx.read_partial() == oracle.sum_range(d, f, k0, k1, 3), (f, d, k0, k1)


@pytest.mark.parametrize("bits", [47, 48, 49, 52, 57, 61])
@pytest.mark.parametrize("m", KINDS)
def test_sums_around_powers_of_two(ctx192, oracle, m, bits):
    for f in (1, 4):
        k = (m - oracle.DEN1[f] + oracle.DEN0[f] - 1) // oracle.DEN0[f]
        for lift in (-1000, 1000, (3 << (bits - 2)) // 7):     # 10 (d - k) around 2^bits, and above
            d = min(k + ((1 << bits) + lift) // 10, D_MAX)
            check(ctx192, oracle, f, d, k, k + 64 * 5 + 17)


@pytest.mark.parametrize("m", KINDS + [(1 << 60) + 1])
def test_groups_across_a_prefix_boundary(ctx192, oracle, m):
    for f, d in ((0, D_MAX), (3, D_MAX - 2)):
        k = (m - oracle.DEN1[f] + oracle.DEN0[f] - 1) // oracle.DEN0[f]
        while (10 * (d - k) + 142) % (1 << 16) > 640:
            k += 1
        for shift in range(0, 64, 9):
            check(ctx192, oracle, f, d, k - shift, k - shift + 700)
