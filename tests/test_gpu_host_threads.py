"""Calls from two host threads at once (tests/native/host_threads_check.cpp over the C-ABI, so that no
interpreter lock keeps the launches apart). Plans of one band shape share their kernels, and a kernel's
shared-memory limit on a device is one for all threads: tiles of very different sizes have to launch
whatever the other thread launches in between."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path_factory.mktemp("threads") / "host_threads_check")
    lib = os.path.join(ROOT, "ddc_b200")
    cmd = ["g++", "-std=c++17", "-O1", "-pthread", "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "native", "host_threads_check.cpp"),
           "-L" + lib, "-lddcb", "-Wl,-rpath," + lib, "-L/usr/local/cuda/lib64", "-lcudart", "-Wl,-rpath,/usr/local/cuda/lib64", "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("small,large,refined", [
    ((300, 16), (1024, 2400), 0),   # one kernel, plans of two sizes
    ((1024, 16), (1024, 2400), 0),  # one plan size, a short and a long batch
    ((600, 64), (1000, 64), 1),     # two tile sizes of the refined solve
])
def test_two_threads(program, small, large, refined):
    args = [*small, *large, 20000, refined]
    r = subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
