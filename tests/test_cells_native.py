"""Cells of non-finite and extreme coordinates (tests/native/cells_check.cpp, on the host, no GPU): inside
the basis whatever the coordinate, so that no kernel indexes outside its tile."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_cells_of_any_coordinate(tmp_path):
    exe = str(tmp_path / "cells_check")
    cmd = ["g++", "-std=c++17", "-O1", "-x", "c++", os.path.join(ROOT, "tests", "native", "cells_check.cpp"), "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and ", 0 failures" in r.stdout, r.stdout
