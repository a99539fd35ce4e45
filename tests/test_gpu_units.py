"""Small checks of the library's internal functions on the GPU, compiled here with nvcc from the headers."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_tiles_cpu import _nvcc

pytestmark = pytest.mark.gpu


def _run(name, tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / name
    cmd = [nvcc, "-std=c++17", "-O2", "-fmad=false", "-gencode", "arch=compute_100a,code=sm_100a",
           "-I", os.path.join(ROOT, "srsoriginal_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", name + ".cu"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)


def test_wave_slots_of_several_block_sizes(tmp_path):
    r = _run("wave_slots_check", tmp_path)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


def test_own_roots_reciprocals_and_sines(tmp_path):
    r = _run("device_math_check", tmp_path)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
