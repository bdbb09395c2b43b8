"""Cell counts of the grids across collimated sources (hrt_device.cuh sun_cells): the shipped header
compiled for the host; a grid never has more cells than its buffer."""
import os
import subprocess

import pytest

from test_fastdiv import _nvcc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not available")
def test_grid_cells_fit_their_buffer(tmp_path):
    exe = str(tmp_path / "suncells_check")
    src = os.path.join(ROOT, "tests", "cpp", "suncells_check.cu")
    r = subprocess.run([_nvcc(), "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "helios_gb300", "csrc"), src, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "failures 0" in r.stdout
