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


@pytest.mark.parametrize("pos", [[5, 1000, 10 ** 6], [17, 2 * 10 ** 10, 10 ** 9 + 7, 300]])
def test_calls_in_a_row_and_captured(cbl, pos):
    """Calls enqueued behind one another (each empties the sums of the one before) and the
    same call replayed from a graph; the second set has tiles of every kind below 2^44."""
    import torch
    fn = cbl.load().cbl_batch_noalloc
    fn.argtypes = [ctypes.POINTER(ctypes.c_uint64), ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    torch.cuda.set_device(0)
    n = len(pos)
    outs = [torch.zeros((n, 3), dtype=torch.int64, device="cuda") for _ in range(4)]

    def call(values, out):
        stream = torch.cuda.current_stream().cuda_stream
        assert fn((ctypes.c_uint64 * n)(*values), n, out.data_ptr(), stream) == 0

    call(pos, outs[0])
    call(pos[::-1], outs[1])
    call(pos, outs[2])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(pos, outs[3])
    for _ in range(2):
        outs[3].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[3], outs[0])
    assert torch.equal(outs[2], outs[0]) and torch.equal(outs[1].flip(0), outs[0])
    w = [int(x) & ((1 << 64) - 1) for x in outs[0].flatten().tolist()]
    with cbl.Context(0, 1) as ctx:
        assert [(w[3 * i] << 128) | (w[3 * i + 1] << 64) | w[3 * i + 2] for i in range(n)] == ctx.batch(pos)
