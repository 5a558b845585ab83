"""The encode kernel against the oracle's encoder, word for word: partial blocks
on every face, rows that allow 16-byte loads and rows that do not, warps with
few blocks, every length of a block's row, and values at the ends of the range."""
import numpy as np
import pytest

import bcmc

pytestmark = pytest.mark.gpu


def _field(dims, kind):
    rs = np.random.default_rng(sum(dims))
    X, Y, Z = dims
    if kind == "smooth":
        z, y, x = np.meshgrid(*(np.arange(n) for n in (Z, Y, X)), indexing="ij")
        f = np.sin(0.3 * x) * np.cos(0.2 * y) + 0.1 * z
    elif kind == "noise":
        f = rs.standard_normal((Z, Y, X))
    else:  # magnitudes from denormal to 3e38, zero blocks, constant blocks
        f = rs.standard_normal((Z, Y, X)) * 10.0 ** rs.integers(-44, 38, (Z, Y, X))
        f[: Z // 2, : Y // 2, : X // 3] = 0.0
        f[:, Y // 2 :, : X // 3] = 3.0
    return np.ascontiguousarray(np.clip(f, -3e38, 3e38).astype(np.float32))


@pytest.mark.parametrize("dims", [(1, 1, 1), (4, 4, 4), (2, 3, 6), (5, 6, 7), (64, 20, 12), (65, 19, 13), (130, 33, 10)])
@pytest.mark.parametrize("kind", ["smooth", "noise", "ends"])
def test_encode(ctx, oracle, dims, kind):
    import torch

    f = _field(dims, kind)
    nb = int(np.prod([(d + 3) // 4 for d in dims]))
    for rate in (1, 2, 3, 4, 7, 13, 16, 31, 32):
        ref = oracle.zfp_encode(f, rate)
        for off in (0, 1):  # a base on a 16-byte boundary, and one off it
            buf = torch.zeros(f.size + 4, dtype=torch.float32, device="cuda")
            buf[off : off + f.size] = torch.from_numpy(f.reshape(-1)).cuda()
            dev = buf[off : off + f.size].view(*f.shape)
            got = bcmc.zfp_encode(ctx, dev, rate)
            got = got.cpu().numpy().view(np.uint64)
            assert np.array_equal(got[: nb * rate], ref[: nb * rate]), (rate, off)
            assert got[nb * rate] == 0
