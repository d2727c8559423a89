"""Registers of the adjoint column passes at lengths whose factors make a thread's state
large, from the compiler's figures (-Xptxas -v): nothing spills, and lengths 168 and 288
keep the three CTAs of 128 threads per SM that 168 registers allow."""
from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    return None


def test_no_spills(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not available")
    r = subprocess.run([nvcc, "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-Xptxas", "-v",
                        "-gencode", "arch=compute_103a,code=sm_103a", "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "opencliper_gb300", "csrc"), "-c",
                        os.path.join(ROOT, "tests", "cpp", "column_registers.cu"), "-o", str(tmp_path / "o.o")],
                       check=True, capture_output=True, text=True)
    seen, kernel, spill = {}, None, 0
    for line in (r.stdout + r.stderr).splitlines():
        if m := re.search(r"Compiling entry function '\w*k_(inv|adj)_colsILi(\d+)ELb(\d)E", line):
            kernel = (m[1], int(m[2]), int(m[3]))
        elif m := re.search(r"(\d+) bytes spill stores", line):
            spill = int(m[1])
        elif kernel and (m := re.search(r"Used (\d+) registers", line)):
            seen[kernel] = (int(m[1]), spill)
            kernel = None
    assert len(seen) == 11, seen
    assert {k: v for k, v in seen.items() if v[1] > 0} == {}
    assert all(seen["inv", n, u][0] <= 168 for n in (168, 288) for u in (0, 1)), seen
