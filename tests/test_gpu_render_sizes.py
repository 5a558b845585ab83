"""The rasteriser's two ways of drawing a triangle, against the oracle: random
triangles from under a pixel to hundreds across, around the box and the side
where one gives way to the other, slivers, and vertices of different blocks."""
import numpy as np
import pytest

from bcmc import camera
from test_gpu_render import _check

pytestmark = pytest.mark.gpu

DIMS = (64, 64, 64)


def _soup(n, spread, seed):
    """n triangles: a random block each, or (spread) a random block per vertex."""
    rng = np.random.default_rng(seed)
    v = np.zeros((3 * n, 2), np.uint32)
    v[:, 0] = rng.integers(0, 1 << 30, 3 * n)
    ids = rng.integers(0, 16**3, n)
    v[:, 1] = np.repeat(ids, 3) if not spread else np.clip(np.repeat(ids, 3) + rng.integers(-1, 2, 3 * n), 0, 16**3 - 1)
    thin = rng.random(n) < 0.2  # two corners alike but for one step
    v[1::3][thin] = v[0::3][thin]
    v[1::3][thin, 0] ^= 1 << 20
    return v


@pytest.mark.parametrize("size", [(37, 23), (160, 120), (640, 480), (1500, 1100)])
@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("fog", [False, True])
def test_soup(ctx, oracle, size, spread, fog):
    w, h = size
    proj, eye = camera.default_view(w, h, eye=(0.2, 0.1, 1.3))
    _check(ctx, oracle, _soup(700, spread, w + spread), DIMS, proj, eye, w, h, (1.0, 0.8, 1.1), fog)
