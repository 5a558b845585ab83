"""bcmc_select_ids into the flags' own words: sizes either side of where a CTA's
range becomes two tiles (8192 elements to a tile, three CTAs an SM), and many."""
import ctypes as C

import numpy as np
import pytest

from bcmc import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("tiles,more", [(0, 1), (1, 0), (1.5, 0), (3, 0), (3, 1), (7.2, 5)])
def test_ids_over_their_flags(ctx, tiles, more, off):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = int(tiles * sms * 8192) + more
    rng = np.random.default_rng(n + off)
    flags = np.where(rng.random(n) < 0.6, rng.integers(1, 1 << 31, n), 0).astype(np.int32)
    buf = torch.zeros(n + off, dtype=torch.int32, device="cuda")
    buf[off:] = torch.from_numpy(flags).cuda()
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = C.c_void_p(buf.data_ptr() + 4 * off)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert _lib.load().bcmc_select_ids(ctx.handle, n, p, p, C.c_void_p(count.data_ptr()), s) == 0
    torch.cuda.synchronize()
    want = np.flatnonzero(flags).astype(np.int32)
    assert int(count.item()) == want.size
    assert np.array_equal(buf[off: off + want.size].cpu().numpy(), want)
