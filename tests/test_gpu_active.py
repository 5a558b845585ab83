"""The active test on words of 32 blocks (k_query_flags, k_active_words) against
the oracle's (compute_block_active.comp:24-61), where rows are shorter than a
word, end inside one, or fill it, at ends of words and of a warp's run of them."""
import numpy as np
import pytest

import bcmc

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (1, 1, 70), (1, 40, 1), (2, 3, 5), (31, 3, 3), (32, 2, 2), (33, 5, 4), (64, 64, 3), (100, 7, 9),
         (4, 4, 64), (129, 33, 17), (300, 300, 20)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("spread", [0.02, 0.4])
def test_block_active(ctx, oracle, grid, spread):
    import torch

    nb = int(np.prod(grid))
    dims = tuple(4 * g for g in grid)
    rng = np.random.default_rng(nb)
    lo = rng.random(nb).astype(np.float32)
    hi = lo + (rng.random(nb) * spread).astype(np.float32)
    ranges = np.stack([lo, hi], 1).reshape(-1).astype(np.float32)
    for iso in (0.01, 0.5, float(lo[nb // 2])):
        got = bcmc.block_active(ctx, torch.from_numpy(ranges).cuda(), dims, iso).cpu().numpy()
        assert np.array_equal(got.astype(np.uint32), oracle.block_active(ranges, dims, iso).astype(np.uint32))
