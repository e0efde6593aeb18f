"""Host-side checks of code that the kernels share with the host (nvcc-compiled, run on
the CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def run(name, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / name)
    r = subprocess.run([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-diag-suppress", "177",
                        "-o", exe, os.path.join(HERE, "cpp", name + ".cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_items_of_lane_groups(tmp_path):
    """Points by groups of lanes: the index of a thread's point where points times lanes
    passes 2^31 (134 million points with 16 lanes)."""
    run("test_group_item", tmp_path)
