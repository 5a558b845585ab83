"""What the engine's autotuner times (csrc/engine_tuning.h), compiled as host C++:
every compiled CTA size of the MC kernel but the one it has timed already, and no
two configurations that launch the same grid."""
import ctypes
import os
import shlex
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib():
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    out = os.path.join(build, "libengine_tuning_host.so")
    cmd = [cxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "webgpu-bcmc_gb300", "csrc"),
           os.path.join(HERE, "host_device", "engine_tuning_host.cpp"), "-o", out]
    cmd += shlex.split(os.environ.get("BCMC_HOST_CXXFLAGS", ""))
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def _list(f, *args):
    out = (ctypes.c_int * 8)()
    return list(out[: f(*args, out)])


@pytest.mark.parametrize("best", [8, 16, 32])
def test_every_other_size(lib, best):
    assert lib.default_size() in (8, 16, 32)
    assert sorted(_list(lib.sizes, best) + [best]) == [8, 16, 32]


@pytest.mark.parametrize("size", [8, 16, 32])
@pytest.mark.parametrize("resident", range(1, 13))
def test_no_grid_twice(lib, size, resident):
    grids = [lib.ctas(size, n, resident) for n in [6] + _list(lib.per_sm, size, resident)]
    assert len(set(grids)) == len(grids)
    assert set(grids) == {lib.ctas(size, n, resident) for n in (4, 5, 6)}
