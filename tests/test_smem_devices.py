"""Kernels that need more than 48 KB of shared memory are opted in on every device that
launches them: the launcher built against a stand-in for the CUDA runtime."""
from __future__ import annotations

import subprocess

from test_problem_memory import _host_program


def test_shared_memory_opt_in_per_device(tmp_path):
    r = subprocess.run([_host_program(tmp_path, "smem_devices")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
