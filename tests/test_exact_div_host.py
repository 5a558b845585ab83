"""exact_div (csrc/exact_div.cuh), compiled as host C++, against the quotient:
every packed position on an axis of every size up to 1200, and of some far above."""
import ctypes
import os
import shlex
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_every_position():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    out = os.path.join(build, "libexact_div_host.so")
    # -ffp-contract=off: only the fused operations that the code names
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "host_device"),
           "-I", os.path.join(ROOT, "webgpu-bcmc_gb300", "csrc"), os.path.join(HERE, "host_device", "exact_div_host.cpp"),
           "-o", out]
    cmd += shlex.split(os.environ.get("BCMC_HOST_CXXFLAGS", ""))
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(out)
    lib.differing.argtypes = [ctypes.c_uint32]
    lib.differing.restype = ctypes.c_uint64
    sizes = list(range(1, 1201)) + [4095, 4096, 65537, 1000003, (1 << 24) - 1]
    with ThreadPoolExecutor(8) as ex:
        bad = [(d, n) for d, n in zip(sizes, ex.map(lib.differing, sizes)) if n]
    assert not bad, bad[:5]
