"""The column-pair iteration's per-length shapes (rowpair.cuh), which nearly every length
runs, checked on the host: a small program built with nvcc prints them.  Every layout
fits a CTA's 227 KB; the CTAs that shared memory lets share an SM never need more than
its 512 tensor-memory columns, so that an allocation never waits on a co-resident CTA of
the same kernel; the launch bound asks for no more CTAs than shared memory holds; a warp
holds whole columns; and the row capacity covers every Cartesian mask at R >= 4."""
from __future__ import annotations

import os
import subprocess

import pytest

from tests.test_rowlocal_shapes import ROOT, _nvcc


def test_pair_shape_rules(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = tmp_path / "pair_shapes"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "opencliper_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "pair_shapes.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(int(v) for v in line.split()) for line in out.splitlines() if line.strip()]
    from tests.test_nesta_gpu import LENGTHS, THREE_PASS_ONLY
    assert {r[0] for r in rows} == set(LENGTHS) - THREE_PASS_ONLY - {280, 360, 392}
    for H, PA, PB, NP, nbytes, bound, tcols, rcap in rows:
        ctas = (228 * 1024) // (nbytes + 1024)
        assert PA * PB == H and PB * NP == 32, H
        assert nbytes <= 227 * 1024 and ctas >= bound, H
        assert tcols * ctas <= 512, H
        assert tcols == 0 or tcols >= 4 * PA, H
        assert rcap >= H // 4 and rcap >= min(H, 32), H
