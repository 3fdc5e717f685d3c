"""The autotuner's cache: entries measured for other kernels are not taken, its own are."""
import pytest

pytestmark = pytest.mark.gpu


def fnv1a(data: bytes) -> int:
    h = 1469598103934665603
    for b in data:
        h = (h ^ b) * 1099511628211 % (1 << 64)
    return h


def test_entries_of_other_kernels_are_measured_again(cbl, tmp_path, monkeypatch):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("CBL_TUNE_CACHE", str(cache))
    pos = [1000, 123455]
    with cbl.Context(0, 1) as ctx:
        want = ctx.batch(pos)
        ctx.set_tuning(2048, 1)
        sms = ctx.prepared_info()["grid"]
        # as stored while the key held the device, its SM count and the positions alone
        old = "%s|sm%d|n%d|h%016x" % (ctx.device_name.replace(" ", "_"), sms, len(pos),
                                      fnv1a(b"".join(p.to_bytes(8, "little") for p in pos)))
        cache.write_text("%s 65536 1\n" % old)
        tile, ctas, ms = ctx.autotune(pos)
        assert ms > 0 and tile != 65536
    with cbl.Context(0, 1) as ctx:
        assert ctx.autotune(pos) == (tile, ctas, -1.0)
        assert ctx.batch(pos) == want


def test_a_cached_choice_leaves_the_positions_prepared(cbl, tmp_path, monkeypatch):
    monkeypatch.setenv("CBL_TUNE_CACHE", str(tmp_path / "tune.txt"))
    pos = [1000, 123455]
    with cbl.Context(0, 1) as ctx:
        ctx.autotune(pos)
    with cbl.Context(0, 1) as ctx:
        want = ctx.batch(pos)
        ctx.prepare([5000])
        assert ctx.autotune(pos)[2] == -1.0
        ctx.run_prepared()
        assert ctx.read_results() == want
