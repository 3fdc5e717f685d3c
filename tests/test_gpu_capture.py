"""A caller that captures the context's stream: calls that upload a tile table are refused, as
a replay would copy another table, and the context works on afterwards."""
import pytest

pytestmark = pytest.mark.gpu


def test_table_uploads_are_refused_under_capture(cbl, oracle):
    import torch
    d, f = 39999, 3
    want = oracle.sum_range(d, f, 17, 9001, 3)
    with cbl.Context(0, 1) as ctx:
        ctx.Set0mem()
        ctx.BatchCalc(17, 9001, f, d)
        ctx.wait()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
            graph.capture_begin(capture_error_mode="thread_local")
            codes = []
            for call in (lambda: ctx.BatchCalc(17, 9001, f, d), lambda: ctx.prepare([100000]),
                         lambda: ctx.Sglobal32mtg(0, d, 100, oracle.SIGN[f], oracle.DEN0[f], oracle.DEN1[f])):
                with pytest.raises(cbl.CblError) as e:
                    call()
                codes.append(e.value.code)
            ctx.Ssum()                                      # kernels alone may be captured
            graph.capture_end()
        assert codes == [-4, -4, -4]
        graph.replay()
        torch.cuda.synchronize()
        assert ctx.read_partial() == want
        ctx.Set0mem()
        ctx.BatchCalc(17, 9001, f, d)
        assert ctx.read_partial() == want


def test_a_whole_call_under_capture_leaves_nothing_prepared(cbl, oracle):
    import torch
    with cbl.Context(0, 1) as ctx:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
            graph.capture_begin(capture_error_mode="thread_local")
            with pytest.raises(cbl.CblError):
                ctx.compute(100000)                         # its wait ends the capture
            with pytest.raises(Exception):
                graph.capture_end()
        with pytest.raises(cbl.CblError) as e:
            ctx.run_prepared()
        assert e.value.code == -1
        assert ctx.compute(1000) == "%048x" % oracle.result(oracle.pos_to_d(1000)[0], 0, 3)
