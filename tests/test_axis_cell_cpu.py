"""Host-side check of the cell index of one-axis field maps, positions that are no number among them
(tests/axis_cell_check.cu, compiled here with nvcc and run on the CPU; no GPU is used)."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_tiles_cpu import _nvcc


def test_cells_stay_in_the_map(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "axis_cell_check"
    cmd = [nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
           "-I", os.path.join(ROOT, "srsoriginal_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "axis_cell_check.cu"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
