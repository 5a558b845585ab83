"""Marching cubes where every cell has vertices: the fullest lists, offsets and
windows of the MC kernels.  Random values against the oracle, on grids that give
a warp one block up to whole runs of them; and a checkerboard of 256^3 voxels,
each cell of which has four triangles, whose vertices are known from one block."""
import numpy as np
import pytest

import bcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 4, 4), (8, 5, 4), (20, 16, 16), (40, 36, 36), (64, 64, 60), (130, 120, 110)])
def test_random_values_match_oracle(ctx, oracle, dims):
    f = np.random.default_rng(dims[0]).random(dims[::-1]).astype(np.float32)
    words = oracle.zfp_encode(f, 16)
    ref = oracle.CompressedMarchingCubes(words, 16, dims, initial_cache_fraction=0.5)
    c = bcmc.Context(0, initial_cache_fraction=0.5)
    mc = bcmc.CompressedMarchingCubes(c)
    mc.setCompressedVolume(words, 16, dims)
    eng = bcmc.Engine(c)
    eng.addVolume(words, 16, dims)
    for iso in (0.5, 0.2, 0.93):
        n_ref = ref.compute_surface(iso)
        assert mc.computeSurface(iso) == n_ref
        want = ref.vertices(n_ref)
        assert np.array_equal(mc.copyVertices(), want)
        res = eng.run([(0, iso)])
        assert int(res["num_vertices"][0]) == n_ref
        assert np.array_equal(eng.copyVertices(), want)


def test_checkerboard(ctx):
    import torch

    n = 256
    i = torch.arange(n, device="cuda")
    f = ((i[:, None, None] + i[None, :, None] + i) % 2).float()
    c = bcmc.Context(0, initial_cache_fraction=1.0)
    words = bcmc.zfp_encode(c, f, 32)
    torch.cuda.synchronize()
    mc = bcmc.CompressedMarchingCubes(c)
    mc.setCompressedVolume(words, 32, (n, n, n))
    total = mc.computeSurface(0.5)
    nb = n // 4
    # a block's cells: four along an axis, three at the volume's far faces
    b = torch.arange(nb**3, device="cuda")
    cells = 1
    for k in (b % nb, b // nb % nb, b // nb**2):
        cells = cells * torch.where(k == nb - 1, 3, 4)
    counts = 12 * cells
    assert total == int(counts.sum())
    v = mc.vertexBuffer.torch()
    assert torch.equal(v[:, 1].long(), torch.repeat_interleave(b, counts))
    views = mc.views()
    assert torch.equal(views["vert_offsets"].torch().long(), torch.cumsum(counts, 0) - counts)
    inner = (counts == 768).nonzero().flatten()
    first = torch.cumsum(counts, 0) - counts
    got = v[:, 0][first[inner][:, None] + torch.arange(768, device="cuda")]
    assert bool((got == got[0]).all())
    eng = bcmc.Engine(c)
    eng.addVolume(words.cpu().numpy(), 32, (n, n, n))
    assert int(eng.run([(0, 0.5)])["num_vertices"][0]) == total
    assert torch.equal(eng.vertexBuffer.torch(), v)
