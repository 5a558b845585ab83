"""A sort captured into a CUDA graph, replayed after an active test whose working
words are larger than the sort's buffers and whose status words are fewer: the
graph's buffers are still the context's."""
import ctypes as C

import numpy as np
import pytest

import bcmc
from bcmc import _lib

pytestmark = pytest.mark.gpu


def test_active_test_leaves_the_sorts_buffers(ctx):
    import torch

    L = _lib.load()
    c = bcmc.Context(ctx.device)
    n, dims = 40_000, (400, 400, 400)  # 10 tiles: 640 KB and 2560 status words; 1 M blocks: 1.4 MB and 1956
    rng = np.random.default_rng(5)
    src = torch.from_numpy(rng.integers(0, 1 << 31, n).astype(np.int32)).cuda()
    ids = torch.arange(n, dtype=torch.int32, device="cuda")
    keys, values = torch.empty_like(src), torch.empty_like(ids)

    def sort(stream):
        keys.copy_(src)
        values.copy_(ids)
        assert L.bcmc_sort_pairs_u32(c.handle, C.c_void_p(keys.data_ptr()), C.c_void_p(values.data_ptr()), n, 0,
                                     C.c_void_p(stream.cuda_stream)) == 0

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        sort(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sort(torch.cuda.current_stream())
    want = keys.clone(), values.clone()
    ranges = torch.rand(100 ** 3, 2, device="cuda")
    bcmc.block_active(c, ranges, dims, 0.5)
    room = torch.empty(1 << 20, dtype=torch.int32, device="cuda")  # would take the place of what was freed
    for _ in range(3):
        keys.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(keys, want[0]) and torch.equal(values, want[1])
    del room
