"""The words that the device ZFP codec (csrc/zfp_device.cuh) touches past a block:
its encoder's row and its decoder's input are as long as they say, at every rate,
under the address sanitizer."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_rows_are_long_enough():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    out = os.path.join(build, "zfp_rows_host")
    cmd = [cxx, "-O1", "-g", "-std=c++17", "-ffp-contract=off", "-fsanitize=address", "-I", os.path.join(HERE, "host_device"),
           "-I", os.path.join(ROOT, "webgpu-bcmc_gb300", "csrc"), os.path.join(HERE, "host_device", "zfp_rows_host.cpp"),
           "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0 and "asan" in r.stderr:
        pytest.skip("no address sanitizer")
    assert r.returncode == 0, r.stderr
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0")
    r = subprocess.run([out], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-3000:]
