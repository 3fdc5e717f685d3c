"""Tile tables built on the device (cbl_batch_noalloc) against cbl_batch: every number of
positions that changes the block's scan, ties, and positions around the kind limits."""
import ctypes
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 11, 12, 13, 31, 32, 33, 63, 64])
def test_tables_equal_batch(cbl, n):
    import torch
    fn = cbl.load().cbl_batch_noalloc
    fn.argtypes = [ctypes.POINTER(ctypes.c_uint64), ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    rng = random.Random(n)
    pos = [rng.choice([5, 6, 15, 1000, 67108871, 67108901, rng.randrange(5, 4000), rng.randrange(5, 10 ** 6)])
           for _ in range(n)]
    torch.cuda.set_device(0)
    out = torch.full((3 * n,), -1, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream()
    assert fn((ctypes.c_uint64 * n)(*pos), n, out.data_ptr(), stream.cuda_stream) == 0
    stream.synchronize()
    w = [int(x) & ((1 << 64) - 1) for x in out.cpu().tolist()]
    with cbl.Context(0, 1) as ctx:
        assert [(w[3 * i] << 128) | (w[3 * i + 1] << 64) | w[3 * i + 2] for i in range(n)] == ctx.batch(pos)
