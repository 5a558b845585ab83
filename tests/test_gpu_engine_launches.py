"""The launches that a batch is counted as: its sequence's kernels (begin, active test,
entries, decode, marching cubes, finish; no entries for up to eight tiles, where the
active test makes them), also when they are replayed as a graph."""
import pytest

import bcmc
from bcmc import _lib
from bcmc import datasets as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kernels", [(1, 5), (8, 5), (9, 6), (12, 6)])
def test_a_batch_counts_its_kernels(ctx, oracle, n, kernels):
    L = _lib.load()
    dims = (40, 36, 36)
    eng = bcmc.Engine(ctx, max_batch=16)
    eng.addVolume(oracle.zfp_encode(D.make_field("turbulence", dims, 1), 6), 6, dims)
    qs = [(0, 0.01 * i) for i in range(n)]
    for _ in range(3):  # the first runs grow buffers and go again
        eng.run(qs)
    before = L.bcmc_kernel_launches()
    eng.run(qs)
    assert L.bcmc_kernel_launches() - before == kernels
