"""RadixSorter at the sizes where the passes change their way of placing tiles
(a tile to a CTA with a barrier, or look-back) and the ways the sorted pairs get
back (the last of several passes, or the one pass there is): against a stable
sort in the reference's tie order."""
import numpy as np
import pytest

import bcmc
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

TILE = 4096


def _want(keys, vals, reverse):
    n = len(keys)
    i = np.arange(n)
    if reverse:  # key desc, chunk asc, index desc
        order = np.lexsort((-i, i // 64, ~keys))
    else:  # key asc, chunk desc, index asc
        order = np.lexsort((i, -(i // 64), keys))
    return keys[order], vals[order]


@pytest.mark.parametrize("n", [65, 7 * TILE, 8 * TILE - 1, 8 * TILE - 4095, 9 * TILE + 1, 100 * TILE + 777, 304 * TILE,
                               304 * TILE + 1, 500 * TILE + 3])
@pytest.mark.parametrize("kind", ["wide", "two_bytes", "one_byte", "one_value", "top_byte"])
@pytest.mark.parametrize("reverse", [False, True])
def test_sizes(ctx, n, kind, reverse):
    rs = np.random.default_rng(n)
    keys = {"wide": lambda: rs.integers(0, 1 << 32, n), "two_bytes": lambda: rs.integers(0, 1 << 16, n),
            "one_byte": lambda: rs.integers(0, 200, n), "one_value": lambda: np.full(n, 77),
            "top_byte": lambda: rs.integers(0, 250, n) << 24}[kind]().astype(np.uint32)
    vals = rs.permutation(n).astype(np.uint32)
    k, v = to_dev(keys), to_dev(vals)
    bcmc.RadixSorter(ctx).sort(k, v, n, reverse)
    wk, wv = _want(keys, vals, reverse)
    assert np.array_equal(to_host(k, np.uint32), wk)
    assert np.array_equal(to_host(v, np.uint32), wv)
