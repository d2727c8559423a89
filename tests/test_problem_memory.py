"""Allocation failures of a problem's workspace, on the host: csrc/nesta_host.cu built
against a stand-in for the CUDA runtime (tests/cpp/fake_cudart.cpp) whose allocations fail
one after the other.  No kernel runs."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CPP = os.path.join(ROOT, "tests", "cpp")


def _nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    return None


def _host_program(tmp_path, name):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / name)
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-cudart", "none", "-Xptxas", "-O0",
                    "-gencode", "arch=compute_103a,code=sm_103a", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "opencliper_gb300", "csrc"), "-I", CPP,
                    os.path.join(CPP, name + ".cu"), os.path.join(CPP, "fake_cudart.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


def test_fit_rows_keeps_the_problem_when_memory_runs_out(tmp_path):
    r = subprocess.run([_host_program(tmp_path, "fit_rows")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_row_local_tiles_are_allocated_where_they_are_used(tmp_path):
    r = subprocess.run([_host_program(tmp_path, "tile_memory")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
