"""read_results covers the positions that the context holds, whichever call prepared them."""
import pytest

pytestmark = pytest.mark.gpu


def test_results_follow_the_last_call_that_prepared(cbl):
    many = [1000 + 5 * i for i in range(300)]
    with cbl.Context(0, 1) as ctx:
        with pytest.raises(cbl.CblError) as e:
            ctx.read_results()                              # nothing prepared
        assert e.value.code == -1
        ctx.prepare([1000])
        want = ctx.batch(many)                              # more than the prepare's
        assert ctx.read_results() == want
        ctx.run_prepared()
        assert ctx.read_results() == want
        digits = ctx.compute(100000)                        # fewer
        assert ["%048x" % v for v in ctx.read_results()] == [digits]
        ctx.prepare(many[:7])
        ctx.run_prepared()
        assert ctx.read_results() == want[:7]
