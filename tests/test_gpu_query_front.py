"""A small volume's query front in one launch (k_query_front: flags, active test and
slots by one cluster) against the three kernels that a query with a perf tracker
runs: volumes of one block, of as many words as leave the cluster's CTAs without
work or with a short last share, and either side of the limit; the LRU state over
queries that decode new blocks, grow the cache, find all cached, and find none."""
import numpy as np
import pytest

import bcmc
from bcmc import datasets as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 4, 4), (64, 32, 16), (68, 33, 17), (64, 64, 64), (96, 100, 60), (128, 96, 128), (128, 97, 128)])
@pytest.mark.parametrize("fraction", [0.05, 1.0])
def test_front_matches_kernels(ctx, oracle, dims, fraction):
    f = D.make_field("turbulence", dims, 9)
    words = oracle.zfp_encode(f, 6)
    lo, hi = float(f.min()), float(f.max())
    c = bcmc.Context(ctx.device, initial_cache_fraction=fraction)
    one, three = bcmc.CompressedMarchingCubes(c), bcmc.CompressedMarchingCubes(c)
    for mc in (one, three):
        mc.setCompressedVolume(words, 6, dims)
    for t in (0.9, 0.88, 0.3, 0.5, 2.0, 0.5, 0.45, 0.1, 0.6, 0.62, 0.9):
        iso = float(np.float32(lo + t * (hi - lo)))
        n = one.computeSurface(iso)
        assert n == three.computeSurface(iso, {})
        assert one.stats() == three.stats()
        assert np.array_equal(one.copyVertices(), three.copyVertices())
        a, b = one.lruCache.state(), three.lruCache.state()
        assert a.keys() == b.keys()
        for k in a:
            assert np.array_equal(a[k], b[k]), (iso, k)
