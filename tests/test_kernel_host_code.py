"""Host-side checks of code that the kernels share with the host and of the host code
beside it (compiled here, run on the CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def compile_and_run(cmd, exe):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)


def run_cu(name, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / name)
    compile_and_run([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-diag-suppress", "177",
                     "-o", exe, os.path.join(HERE, "cpp", name + ".cu")], exe)


def test_items_of_lane_groups(tmp_path):
    """Points by groups of lanes: the index of a thread's point where points times lanes
    passes 2^31 (134 million points with 16 lanes)."""
    run_cu("test_group_item", tmp_path)


def test_pinned_memory_is_optional(tmp_path):
    """A handle's page-locked memory: refused in full, it is created with the part that it
    needs (the parameters then take the copies of large problems)."""
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    exe = str(tmp_path / "test_pinned")
    compile_and_run([gxx, "-O1", "-std=c++17", "-Wall", "-Wextra", "-o", exe, os.path.join(HERE, "cpp", "test_pinned.cpp")],
                    exe)
