"""The launches that a batch is counted as: its sequence's kernels (begin, active test,
entries, decode, marching cubes, finish), also when they are replayed as a graph."""
import pytest

import bcmc
from bcmc import _lib
from bcmc import datasets as D

pytestmark = pytest.mark.gpu


def test_a_batch_counts_its_kernels(ctx, oracle):
    L = _lib.load()
    dims = (40, 36, 36)
    eng = bcmc.Engine(ctx, max_batch=16)
    eng.addVolume(oracle.zfp_encode(D.make_field("turbulence", dims, 1), 6), 6, dims)
    qs = [(0, 0.01 * i) for i in range(12)]
    for _ in range(3):  # the first runs grow buffers and go again
        eng.run(qs)
    before = L.bcmc_kernel_launches()
    eng.run(qs)
    assert L.bcmc_kernel_launches() - before == 6
