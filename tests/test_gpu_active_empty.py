"""bcmc_block_active on a volume without blocks: nothing to test, and no error."""
import ctypes as C

import pytest

from bcmc import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(0, 8, 8), (8, 0, 8), (8, 8, 0), (0, 0, 0)])
def test_no_blocks(ctx, dims):
    import torch

    ranges = torch.zeros(16, device="cuda")
    active = torch.full((8,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = _lib.load().bcmc_block_active(ctx.handle, C.c_void_p(ranges.data_ptr()), (C.c_uint32 * 3)(*dims), C.c_float(0.5),
                                       C.c_void_p(active.data_ptr()), None)
    assert st == 0
    ctx.synchronize()
    assert active.tolist() == [7] * 8
