"""bcmc_memory_report's total against what the context counts as allocated: after a
volume's load, after queries that grow its cache and vertex buffer, and after a
sweep into host memory, which adds vertex buffers."""
import ctypes as C

import numpy as np
import pytest

import bcmc
from bcmc import _lib
from bcmc import datasets as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 4, 4), (64, 64, 64), (130, 97, 61)])
def test_total_is_what_is_held(ctx, oracle, dims):
    import torch

    f = D.make_field("turbulence", dims, 2)
    words = oracle.zfp_encode(f, 4)
    c = bcmc.Context(ctx.device, initial_cache_fraction=0.05)
    counter = bcmc.Engine(c)  # its statistics have the context's device bytes
    before = counter.stats()["device_bytes"]
    mc = bcmc.CompressedMarchingCubes(c)
    mc.setCompressedVolume(words, 4, dims)

    def check():
        m = _lib.bcmc_memory()
        assert _lib.load().bcmc_memory_report(mc._vol, C.byref(m)) == 0
        assert m.deviceTotal == counter.stats()["device_bytes"] - before

    check()
    isos = [float(f.min() + t * (f.max() - f.min())) for t in (0.9, 0.5, 0.2, 0.6, 0.4, 0.55)]
    for iso in isos:
        mc.computeSurface(iso)
        check()
    out = torch.zeros((1 << 23, 2), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    mc.computeSurfacesToHost(isos, out)
    check()
