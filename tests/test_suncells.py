"""Host checks of the shipped headers: a grid across a collimated source never has more cells than its
buffer (sun_cells), and the bounds on ray origins hold the primitives' edges and the walls."""
import os
import subprocess

import pytest

from test_fastdiv import _nvcc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not available")
@pytest.mark.parametrize("check", ["suncells", "reach"])
def test_host_check(tmp_path, check):
    exe = str(tmp_path / check)
    src = os.path.join(ROOT, "tests", "cpp", check + "_check.cu")
    r = subprocess.run([_nvcc(), "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "helios_gb300", "csrc"), src, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "failures 0" in r.stdout
