"""Host-side check of the plans callers get without options (tests/native/default_plan_check.cpp, no
GPU): degrees 1-5, uniform, perturbed and graded meshes, five closure pairs, sizes around the multiples
of a chunk's rows and around the longest lines of the register solve, FP64 and refined builders."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_default_plans(tmp_path):
    exe = str(tmp_path / "default_plan_check")
    cmd = ["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-x", "c++",
           os.path.join(ROOT, "ddc_b200", "csrc", "plan.cpp"), os.path.join(ROOT, "tests", "native", "default_plan_check.cpp"),
           "-x", "none", "-L/usr/local/cuda/lib64", "-lcudart", "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and " 0 failures" in r.stdout, r.stdout[-3000:]
