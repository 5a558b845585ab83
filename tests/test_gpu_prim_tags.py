"""The primitives of one context share its status words, which a sort of more tiles
than run at once leaves with the tags of its passes: the scans, selects and active
tests that follow, at every distance, take none of them for their own.  (A wrong tag
shows only when a CTA reads a word before its owner has written it: this holds the
sequences that could go wrong to their results, it does not force that order.)"""
import ctypes as C

import numpy as np
import pytest

import bcmc
from bcmc import _lib
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["scan", "select", "active"])
def test_after_a_long_sort(ctx, oracle, kind):
    import torch

    c = bcmc.Context(ctx.device)
    L = _lib.load()
    rs = np.random.default_rng(3)
    n = 400 * 4096 + 9
    keys = rs.integers(0, 1 << 32, n).astype(np.uint32)
    dims = (128, 128, 128)
    lo = rs.random(32**3).astype(np.float32)
    ranges = np.stack([lo, lo + np.float32(0.05)], 1).reshape(-1).astype(np.float32)
    active = oracle.block_active(ranges, dims, 0.5).astype(np.uint32)
    for op in range(12):
        if op in (0, 2):  # the passes of the first and third operation: tags 4 to 7 and 12 to 15
            k, v = to_dev(keys), to_dev(np.arange(n, dtype=np.uint32))
            bcmc.RadixSorter(c).sort(k, v, n, False)
            assert np.array_equal(to_host(k, np.uint32), np.sort(keys))
        elif kind == "active":
            got = bcmc.block_active(c, torch.from_numpy(ranges).cuda(), dims, 0.5).cpu().numpy()
            assert np.array_equal(got.astype(np.uint32), active), op
        else:
            m = 200_000 + op
            a = (rs.random(m) < 0.4).astype(np.uint32)
            d, out = to_dev(a), torch.zeros(m, dtype=torch.int32, device="cuda")
            tot = torch.zeros(1, dtype=torch.int32, device="cuda")
            f = L.bcmc_scan_exclusive_u32_async if kind == "scan" else L.bcmc_select_ids
            args = (d.data_ptr(), out.data_ptr(), m) if kind == "scan" else (m, d.data_ptr(), out.data_ptr())
            torch.cuda.synchronize()
            assert f(c.handle, *args, tot.data_ptr(), C.c_void_p(1)) == 0
            torch.cuda.synchronize()
            total = int(a.sum())
            assert int(tot[0]) == total, op
            got = to_host(out, np.uint32)
            if kind == "scan":
                assert np.array_equal(got, np.cumsum(a, dtype=np.uint32) - a), op
            else:
                assert np.array_equal(got[:total], np.flatnonzero(a).astype(np.uint32)), op
