"""The share-out of the LRU's slots (csrc/slot_ranges.cuh), compiled as host C++:
the CTAs that publish a count each have a status word of the slots' own, for
k_query_front's sixteen CTAs over caches from one chunk on as for k_slots' grids."""
import ctypes
import os
import shlex
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    out = os.path.join(build, "libslot_ranges_host.so")
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(HERE, "host_device"),
           "-I", os.path.join(ROOT, "webgpu-bcmc_gb300", "csrc"), os.path.join(HERE, "host_device", "slot_ranges_host.cpp"),
           "-o", out]
    cmd += shlex.split(os.environ.get("BCMC_HOST_CXXFLAGS", ""))
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(out)
    lib.check_ranges.argtypes = [ctypes.c_uint32, ctypes.c_uint32]
    return lib.check_ranges


@pytest.mark.parametrize("ctas", [1, 2, 16, 608])
def test_publishing_ctas_have_a_status_word(check, ctas):
    sizes = list(range(32, 26000, 32)) + [2_600_000, (1 << 31) - 32, 0xffffffe0]
    assert not [(s, e) for s in sizes if (e := check(s, ctas))]
