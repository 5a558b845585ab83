"""The scan, the fused select and the compaction at the ends of tiles and of a
CTA's range of tiles, with arrays on 16-byte boundaries and off them."""
import ctypes as C

import numpy as np
import pytest

import bcmc
from bcmc import _lib

pytestmark = pytest.mark.gpu

TILE = 8192


@pytest.mark.parametrize("n", [1, 15, 16, 17, TILE - 1, TILE, TILE + 1, 3 * TILE + 5, 456 * TILE, 456 * TILE + 1, 1300 * TILE - 7])
@pytest.mark.parametrize("off", [0, 1])
def test_scan_select_compact(ctx, n, off):
    import torch

    L = _lib.load()
    rs = np.random.default_rng(n)
    a = rs.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    a[rs.random(n) < 0.6] = 0
    want = np.concatenate([np.zeros(1, np.uint64), np.cumsum(a, dtype=np.uint64)]).astype(np.uint32)  # mod 2^32

    def dev(x, extra=8):
        b = torch.zeros(len(x) + extra, dtype=torch.int32, device="cuda")
        b[off : off + len(x)] = torch.from_numpy(x.view(np.int32)).cuda()
        return b, C.c_void_p(b.data_ptr() + 4 * off)

    data, p = dev(a)
    tot = C.c_uint32()
    torch.cuda.synchronize()
    assert L.bcmc_scan_exclusive_u32(ctx.handle, p, n, n + 4, C.byref(tot)) == 0
    assert tot.value == int(want[n])
    assert np.array_equal(data[off : off + n + 1].cpu().numpy().view(np.uint32), want)

    flags, pf = dev(a)
    out, po = dev(np.zeros(n, np.uint32))
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert L.bcmc_select_ids(ctx.handle, n, pf, po, C.c_void_p(count.data_ptr()), None) == 0
    ctx.synchronize()
    ids = np.flatnonzero(a).astype(np.uint32)
    assert int(count[0]) == len(ids)
    assert np.array_equal(out[off : off + len(ids)].cpu().numpy().view(np.uint32), ids)

    rank = np.concatenate([[0], np.cumsum(a != 0)[:-1]]).astype(np.uint32)
    offs, pr = dev(rank)
    out2, p2 = dev(np.zeros(n, np.uint32))
    torch.cuda.synchronize()
    assert L.bcmc_compact_ids(ctx.handle, n, pf, pr, p2, None) == 0
    ctx.synchronize()
    assert np.array_equal(out2[off : off + len(ids)].cpu().numpy().view(np.uint32), ids)
