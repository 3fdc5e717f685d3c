"""The host's launch rules (csrc/cbl_internal.h), compiled for the CPU: how a pass is
dealt out to blocks."""
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
