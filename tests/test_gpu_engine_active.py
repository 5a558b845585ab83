"""The batched engine's active test and entry list, whose words of 32 blocks are
tested with the rows around them: rows of one block, of a word and a block, of
the longest that are read with their neighbours and of the next length; volumes
of less than a tile of 1024 blocks and of several.  Counts, entries and vertices
of every query against the per-query path."""
import numpy as np
import pytest

import bcmc
from bcmc import datasets as D

pytestmark = pytest.mark.gpu

DIMS = [(4, 4, 4), (4, 4, 5000), (130, 20, 36), (132, 68, 40), (1024, 16, 20), (1028, 16, 20), (2060, 4, 9), (128, 128, 128)]


@pytest.mark.parametrize("dims", DIMS)
def test_engine_entries_match_query(ctx, oracle, dims):
    f = D.make_field("turbulence", dims, 4)
    words = oracle.zfp_encode(f, 8)
    lo, hi = float(f.min()), float(f.max())
    isos = [float(np.float32(lo + t * (hi - lo))) for t in (0.5, 0.08, 0.3, 0.97, 1.5, 0.7)]
    mc = bcmc.CompressedMarchingCubes(ctx)
    mc.setCompressedVolume(words, 8, dims)
    eng = bcmc.Engine(ctx)
    a = eng.addVolume(words, 8, dims)
    b = eng.addVolume(words, 8, dims)
    res = eng.run([(v, iso) for iso in isos for v in (a, b)])
    verts = eng.copyVertices()
    for i, iso in enumerate(isos):
        n = mc.computeSurface(iso)
        want = mc.copyVertices()
        active = mc.stats()["numActiveBlocks"]
        for k, r in enumerate(res[2 * i: 2 * i + 2]):
            if n:  # a query without active blocks leaves the statistics of the one before
                assert int(r["num_active_blocks"]) == active, (iso, k)
            assert int(r["num_vertices"]) == n
            off = int(r["vertex_offset"])
            assert np.array_equal(verts[off: off + n], want)
