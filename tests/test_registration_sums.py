"""Where the one-launch registration descent keeps its partial sums of Dif^2
(csrc/reg_sums.h): a CTA that is late into a phase must not read sums that others
store in the same phase.  The phases' order is modelled on the host; the late CTA is
not provoked on a GPU."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_late_block_reads_its_own_iteration(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "reg_sums"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "opencliper_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "reg_sums.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
