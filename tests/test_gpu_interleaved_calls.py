"""Kernel-by-kernel calls between a prepare and its passes, and passes between
kernel-by-kernel calls: neither changes what the other sums."""
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def job(ctx, oracle, d, f, k0, k1):
    ctx.Set0mem()
    ctx.BatchCalc(k0, k1, f, d)
    assert ctx.read_partial() == oracle.sum_range(d, f, k0, k1, 3)


@pytest.mark.parametrize("graph", [True, False])
def test_prepared_passes_around_jobs(cbl, oracle, graph):
    g = load_golden("oracle_small.json")
    pos = [1000, 1000000, 100000]
    want = [int(g[str(p)]["hex192"], 16) for p in pos]
    with cbl.Context(0, 1) as ctx:
        ctx.set_graph(graph)
        ctx.prepare(pos)
        job(ctx, oracle, 3999999999, 2, 429400000, 429470000)
        for _ in range(2):
            ctx.run_prepared()
            assert ctx.read_results() == want
            job(ctx, oracle, 39999, 5, 3, 30001)
            ctx.Sum7(4)
        # the position that a whole call leaves prepared, its shift included
        digits = ctx.compute_hexpos(123457)
        job(ctx, oracle, 39999, 0, 1, 2)
        ctx.run_prepared()
        assert "%048x" % ctx.read_results()[0] == digits


def test_budgeted_pass_around_jobs(cbl, oracle):
    big = load_golden("oracle_big.json")
    with cbl.Context(0, 1) as ctx:
        ctx.prepare([10 ** 9])
        done, total = ctx.run_prepared_budget(4.0)
        assert 0 < done < total
        while done < total:
            job(ctx, oracle, 39999, 3, 17, 9001)
            blob = ctx.checkpoint()
            ctx.prepare([10 ** 9])
            ctx.restore(blob)
            job(ctx, oracle, 3999999999, 2, 429400000, 429420000)
            done, total = ctx.run_prepared_budget(10.0)
        assert "%048x" % ctx.read_results()[0] == big["1000000000"]["hex192"]


def test_sums_around_prepared_passes(cbl, oracle):
    """bigSum keeps what it holds while positions are prepared, run and computed."""
    d, f = 39999, 6
    with cbl.Context(0, 1) as ctx:
        ctx.prepare([100000])
        ctx.Set0mem()
        ctx.Sglobal64mtg(0, d, 1000, oracle.SIGN[f], oracle.DEN0[f], oracle.DEN1[f])
        ctx.run_prepared()
        ctx.compute(1000)
        ctx.Sglobal64mtg(1000, d, d, oracle.SIGN[f], oracle.DEN0[f], oracle.DEN1[f])
        ctx.Ssum()
        assert ctx.read_partial() == oracle.sum_range(d, f, 0, d, 3)
