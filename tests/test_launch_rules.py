"""The host's launch rules (csrc/cbl_internal.h), compiled for the CPU: how a pass is
dealt out to blocks, and how many flushes a digit-sum slot can take from it."""
import ctypes
import os
import subprocess

import pytest

from clbellard_gb300 import build as B

SOURCE = r"""
#include "cbl_internal.h"
extern "C" void split(uint64_t ntiles, uint32_t tile_k, int grid, uint32_t out[3])
{
    const cbl::TileSplit s = cbl::tile_split(ntiles, tile_k, grid);
    out[0] = s.log2_parts;
    out[1] = s.fixed;
    out[2] = s.part_k;
}
extern "C" uint64_t flushes(uint64_t ntiles, uint32_t tile_k, int grid) { return cbl::flush_bound(ntiles, tile_k, grid); }
extern "C" int blocks(int ctas, int resident) { return cbl::tuned_blocks(ctas, resident); }
extern "C" int block_threads() { return cbl::kBlock192; }
extern "C" int carry(uint64_t n) { return cbl::slot_needs_carry(n); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", B.CSRC, "-I", cuda,
                    str(d / "rules.cpp"), "-o", str(d / "rules.so")], check=True)
    lib = ctypes.CDLL(str(d / "rules.so"))
    lib.split.argtypes = [ctypes.c_uint64, ctypes.c_uint32, ctypes.c_int, ctypes.POINTER(ctypes.c_uint32)]
    lib.flushes.argtypes = [ctypes.c_uint64, ctypes.c_uint32, ctypes.c_int]
    lib.flushes.restype = ctypes.c_uint64
    lib.carry.argtypes = [ctypes.c_uint64]
    return lib


def split(rules, ntiles, tile_k, grid):
    out = (ctypes.c_uint32 * 3)()
    rules.split(ntiles, tile_k, grid, out)
    return tuple(out)


GRIDS = (152, 304, 1064, 1368)
TILES = list(range(32, 1 << 15, 32)) + [65568, 131104, (1 << 20) + 32, (1 << 31) - 32]


@pytest.mark.parametrize("grid", GRIDS)
def test_parts_cover_their_tile(rules, grid):
    """Every term of a tile is in one of its parts, for every tile size that
    cbl_set_tuning takes (multiples of 32), and parts keep whole groups of 64 terms."""
    for tile_k in TILES:
        for ntiles in (1, 2, 7, 85, 2 * grid, 4 * grid - 1):
            log2_parts, fixed, part_k = split(rules, ntiles, tile_k, grid)
            assert fixed == 1
            assert part_k << log2_parts >= tile_k, (tile_k, ntiles)
            assert log2_parts == 0 or part_k % 64 == 0, (tile_k, ntiles)
        assert split(rules, 4 * grid, tile_k, grid) == (0, 0, tile_k)


def flushes_in_shares(segments, tile_k, split, blocks):
    """Flushes of a pass in fixed shares into the one slot of its segments (term counts),
    dealt out as the term kernel does it: a block's items go to its four warps in turn, a
    warp flushes at a change of segment, and the warps still in warp 0's segment at the
    end flush once together."""
    log2_parts, _, part_k = split
    items = []                                              # the segment of each part, None past its end
    for s, n in enumerate(segments):
        for t in range(-(-n // tile_k)):
            items += [s if t * tile_k + p * part_k < min(n, (t + 1) * tile_k) and p * part_k < tile_k else None
                      for p in range(1 << log2_parts)]
    total = 0
    for b in range(blocks):
        share = items[len(items) * b // blocks:len(items) * (b + 1) // blocks]
        last = []
        for w in range(4):
            run = [s for s in share[w::4] if s is not None]
            total += sum(x != y for x, y in zip(run, run[1:]))
            last.append(run[-1] if run else None)
        total += sum(s is not None and s != last[0] for s in last) + (last[0] is not None)
    return total


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("segments", [[65536], [1], [2048 * 3, 20], [100000, 300, 5, 20], [409600]])
def test_flush_bound_covers_fixed_shares(rules, grid, segments):
    for tile_k in (64, 2048, 4128, 65536):
        ntiles = sum(-(-n // tile_k) for n in segments)
        sp = split(rules, ntiles, tile_k, grid)
        bound = rules.flushes(ntiles, tile_k, grid)
        if sp[1]:
            blocks = min(grid, ntiles << sp[0])
            assert flushes_in_shares(segments, tile_k, sp, blocks) <= bound
        else:
            assert bound == ntiles


def test_carry_before_a_digit_sum_can_wrap(rules):
    """Launches of 65,536 terms into one slot, 32 tiles each, make hundreds of flushes a
    launch: the carry is on well before 2^32 of them."""
    sp = split(rules, 32, 2048, 1368)
    made = flushes_in_shares([65536], 2048, sp, min(1368, 32 << sp[0]))
    assert made > 10 * 32
    launches = (1 << 32) // made                            # as many as could not wrap
    assert rules.carry(launches * rules.flushes(32, 2048, 1368))
    assert not rules.carry((1 << 31) - 1)


@pytest.mark.parametrize("resident", [1, 7, 9, 16])
def test_tuning_counts_256_threads_a_cta(rules, resident):
    """A setting of n CTAs is n x 256 threads an SM, up to what is resident."""
    threads = rules.block_threads()
    for ctas in (1, 2, 3, 4, 5, 8, 1000, (1 << 31) - 1):
        assert rules.blocks(ctas, resident) * threads == min(ctas * 256, resident * threads), ctas
    assert rules.blocks(0, resident) == resident
