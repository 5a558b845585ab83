"""The MC kernels' case table and division-free vertex (csrc/mc_triangle.cuh),
compiled as host C++: the table against the entries it is made from, and every
vertex that the fast expression claims against mc_vertex, bit for bit, whichever
way the approximate reciprocal is off, with vertices drawn near the whole numbers
where the two could part."""
import ctypes
import os
import shlex
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(BUILD, "libmc_triangle_host.so")


@pytest.fixture(scope="module")
def lib():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    os.makedirs(BUILD, exist_ok=True)
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "host_device"),
           "-I", os.path.join(ROOT, "webgpu-bcmc_gb300", "csrc"),
           os.path.join(HERE, "host_device", "mc_triangle_host.cpp"), "-o", LIB]
    cmd += shlex.split(os.environ.get("BCMC_HOST_CXXFLAGS", ""))  # e.g. sanitizers
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(LIB)


def test_table(lib):
    for c in range(256):
        n = lib.ref_count(c)
        assert 3 * lib.tri_count(c) == n
        assert [lib.word_entry(c, k) for k in range(n)] == [lib.ref_entry(c, k) for k in range(n)]


@pytest.mark.parametrize("ulps", [-1, 0, 1])
@pytest.mark.parametrize("spread", ["generic", "near", "wild"])
def test_fast_vertex(lib, ulps, spread):
    rng = np.random.default_rng(7 + ulps)
    n = 400_000
    scale = 10.0 ** rng.uniform(-2, 4, n)
    corners = (rng.normal(size=(n, 8)) * scale[:, None]).astype(np.float32)
    iso = (rng.normal(size=n) * scale).astype(np.float32)
    case = ((corners <= iso[:, None]) << np.arange(8)).sum(1).astype(np.uint32)
    keep = (case > 0) & (case < 255)
    corners, iso, case = corners[keep], iso[keep], case[keep]
    n = len(case)
    counts = np.array([lib.ref_count(c) for c in range(256)], np.uint32)
    k = (rng.integers(0, 1 << 30, n) % counts[case]).astype(np.uint32)
    cell = rng.integers(0, 64, n).astype(np.uint32)
    if spread == "near":  # the isovalue where the vertex falls next to a whole number
        e = np.array([[lib.word_entry(c, j) if j < counts[c] else 0 for j in range(15)] for c in range(256)])[case, k]
        off = {0: 0, 1: 1, 5: 2, 6: 3, 25: 4, 26: 5, 30: 6, 31: 7}
        lut = np.array([off.get(i, 0) for i in range(32)])
        fa = corners[np.arange(n), lut[e & 31]].astype(np.float64)
        fb = corners[np.arange(n), lut[(e >> 5) & 31]].astype(np.float64)
        c0 = rng.integers(0, 4, n) * 0.75  # the fractions that the four coordinates leave
        x = rng.integers(0, 256, n) + c0 + rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-6, -2.5, n)
        iso = (fa + np.clip(x / 255.75, 0, 1) * (fb - fa)).astype(np.float32)
    elif spread == "wild":  # ends too close, far apart, infinite and not numbers
        pick = rng.integers(0, 6, n)
        corners[pick == 0] = (iso[pick == 0, None] + rng.choice([-4e-4, 4e-4], (int((pick == 0).sum()), 8))).astype(np.float32)
        corners[pick == 1, ::2] = np.float32(3e38)
        corners[pick == 2, 1::2] = -np.float32(3e38)
        corners[pick == 3, 0] = np.inf
        corners[pick == 4, 3] = np.nan
    fast, exact, again = np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(n, np.uint8)
    corners = np.ascontiguousarray(corners)
    lib.vertices(n, *(a.ctypes.data_as(ctypes.c_void_p) for a in (case, k, cell, corners, iso)), ulps,
                 *(a.ctypes.data_as(ctypes.c_void_p) for a in (fast, again, exact)))
    sure = again == 0
    bad = np.flatnonzero(sure & (fast != exact))
    assert bad.size == 0, (fast[bad[:4]], exact[bad[:4]], corners[bad[:4]], iso[bad[:4]])
    if spread == "generic":
        assert sure.mean() > 0.99
