"""Batches whose queries take one, two and three rounds to find a tile's query among
(32 to a round), and batches of one group of eight tiles (whose entries k_bactive
makes) and of more, over volumes of one tile and of two: the same counts and meshes
as in batches of a few."""
import numpy as np
import pytest

import bcmc
from bcmc import datasets as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,part", [(7, 3), (8, 5), (9, 8), (31, 8), (32, 16), (33, 16), (1024, 16), (1025, 16), (2100, 16)])
def test_batch_equals_its_parts(ctx, oracle, n, part):
    eng = bcmc.Engine(ctx, max_batch=4096)
    for dims in ((12, 8, 8), (56, 44, 40)):
        eng.addVolume(oracle.zfp_encode(D.make_field("blobs", dims, 3), 8), 8, dims)
    rng = np.random.default_rng(n)
    qs = [(int(v), float(np.float32(i))) for v, i in zip(rng.random(n) < 0.1, rng.uniform(0.05, 1.0, n))]
    res = eng.run(qs)
    mesh = eng.copyVertices()
    for a in range(0, n, part):
        got = eng.run(qs[a: a + part])
        assert np.array_equal(got["num_vertices"], res["num_vertices"][a: a + part])
        assert np.array_equal(got["num_active_blocks"], res["num_active_blocks"][a: a + part])
        first = int(res["vertex_offset"][a])
        assert np.array_equal(eng.copyVertices(), mesh[first: first + int(got["num_vertices"].sum())])


def test_one_group_with_a_full_pool(ctx, oracle):
    """Batches of one group whose blocks do not fit the pool beside the last batch's:
    claims run out, slots are evicted, and the batch runs again."""
    dims = (40, 36, 36)  # 810 blocks, one tile
    words = [oracle.zfp_encode(D.make_field("turbulence", dims, s), 6) for s in range(3)]
    small, large = bcmc.Engine(ctx, pool_slots=820), bcmc.Engine(ctx)
    for w in words:
        small.addVolume(w, 6, dims)
        large.addVolume(w, 6, dims)
    for i in range(9):
        q = [(i % 3, 0.05 * (i - 4))] * (1 + i % 2)
        a, b = small.run(q), large.run(q)
        assert np.array_equal(a["num_vertices"], b["num_vertices"]) and a["num_vertices"][0] > 0
        assert np.array_equal(a["num_active_blocks"], b["num_active_blocks"])
        assert np.array_equal(small.copyVertices(), large.copyVertices())
    assert small.stats()["evicted_blocks"] > 0 and large.stats()["evicted_blocks"] == 0
