"""Small passes, cut into parts with one share a block: results equal the oracle for
tile sizes that do and do not divide into 64-term parts, on both sides of one tile a
resident warp, for one and for many positions, with the digit-sum carry on and off."""
import random

import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 0])
@pytest.mark.parametrize("tile", [32, 64, 96, 160, 992, 2048, 65536])
def test_tile_sizes(cbl, tile, ctas):
    g = load_golden("oracle_small.json")
    with cbl.Context(0, 1) as ctx:
        ctx.set_tuning(tile, ctas)
        for p in ("5", "1000", "100000", "1000000", "10000000"):
            if p in g:
                assert ctx.compute(int(p)) == g[p]["hex192"], p


@pytest.mark.parametrize("preset", [None, [(1 << 64) - (1 << 20)] * 6])
def test_counts_around_one_tile_a_warp(cbl, oracle, preset):
    """d chosen so that the tiles of one series pass the number of resident warps."""
    with cbl.Context(0, 1) as ctx:
        ctx.set_tuning(64, 1)
        ctx.prepare([1000])
        warps = ctx.prepared_info()["grid"] * 8
        ctx.set_slot_preset(preset)
        rng = random.Random(warps)
        pos = []
        for tiles in (warps - 9, warps - 1, warps, warps + 1):
            d = tiles * 64 // 7
            pos.append((d * 5 + 3) // 2 + 1 + rng.randrange(30))
        start = sum(v << (32 * j) for j, v in enumerate(preset or [])) * sum((32, 1, 256, 64, 4, 4, 1))
        for p in pos:
            d, _ = oracle.pos_to_d(p)
            assert ctx.batch([p])[0] == (oracle.result(d, 0, 3) + start) % (1 << 192), p


def test_many_short_positions(ctx192, oracle):
    rng = random.Random(7)
    pos = [rng.randrange(5, 3000) for _ in range(300)]
    for p, g in zip(pos, ctx192.batch(pos)):
        assert g == oracle.result(oracle.pos_to_d(p)[0], 0, 3), p
