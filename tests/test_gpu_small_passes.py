"""Small passes with tile sizes that no power of two divides into 64-term parts: whole
calls, prepared passes and one-series ranges keep every term of a tile."""
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [4128, 8224, 12320, 65568])
def test_every_term_of_a_tile(cbl, oracle, tile):
    g = load_golden("oracle_small.json")
    with cbl.Context(0, 1) as ctx:
        ctx.set_tuning(tile)
        for p in (100000, 1000000):
            want = g[str(p)]["hex192"]
            assert ctx.compute(p) == want, p
            ctx.prepare([p])
            ctx.run_prepared()
            assert "%048x" % ctx.read_results()[0] == want, p
        d = 3999999999
        for f, k0, n in ((2, 429400000, 70001), (0, 17, 3 * tile + 1)):
            ctx.Set0mem()
            ctx.BatchCalc(k0, k0 + n, f, d)
            assert ctx.read_partial() == oracle.sum_range(d, f, k0, k0 + n, 3), (f, k0)


def test_tuning_counts_256_threads_a_cta(cbl, oracle):
    """Settings and the reported grid are CTAs of 256 threads: the automatic grid is one
    that an SM's 2048 threads can hold, and no setting changes the bits."""
    g = load_golden("oracle_small.json")
    with cbl.Context(0, 1) as ctx:
        ctx.prepare([1000000])
        auto = ctx.prepared_info()["grid"]
        ctx.set_tuning(2048, 1)
        sms = ctx.prepared_info()["grid"]
        assert sms < auto <= sms * 8
        for ctas in (1, 2, 3, 5, 64):
            ctx.set_tuning(2048, ctas)
            assert ctx.prepared_info()["grid"] == min(ctas * sms, auto)
            assert ctx.compute(1000000) == g["1000000"]["hex192"]
            assert ctx.compute(100000) == g["100000"]["hex192"]
