"""Checkpoints of a large table: the table's identity is formed once, not by every save."""
import random
import time

import pytest

pytestmark = pytest.mark.gpu


def test_later_checkpoints_do_not_hash_the_table_again(cbl):
    rng = random.Random(4096)
    pos = [rng.randrange(1000, 3000) for _ in range(20000)]
    with cbl.Context(0, 1) as ctx:
        ctx.prepare(pos)
        ctx.wait()

        def save():
            t = time.perf_counter()
            blob = ctx.checkpoint()
            return time.perf_counter() - t, blob

        first, blob = save()
        later = [save() for _ in range(5)]
        assert all(b == blob for _, b in later)
        # a full identity is a byte-wise hash of 14 segments of 48 bytes a position; what is left
        # moves 336 bytes a position
        assert min(t for t, _ in later) < first / 2
        ctx.prepare(pos[:-1] + [pos[-1] + 1000])               # another table: another identity
        with pytest.raises(cbl.CblError):
            ctx.restore(blob)
