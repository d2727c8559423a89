"""The FFT process at the lengths whose column pass has a form for few CTAs and one for
many (first factors 17 to 24, and 512), with as many images as the last of the one and
the first of the other take, against the FP64 transform; an image's result does not depend
on how many others there are.  The per-operator bar of test_ops_gpu.py (1e-5; an FFT of
these lengths rounds at ~1e-7), and between the forms twice that rounding."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from opencliper_gb300 import api
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("H", [280, 288, 320, 336, 360, 384, 504, 512])
def test_both_forms(ctx, H):
    W = 24
    line = 3 * torch.cuda.get_device_properties(0).multi_processor_count // (W // 8)  # images of three CTAs
    r = np.random.default_rng(H)
    k = (r.standard_normal((line + 1, 1, H, W)) + 1j * r.standard_normal((line + 1, 1, H, W))).astype(np.complex64)
    for direction, want in ((-1, np.fft.fft2), (1, np.fft.ifft2)):
        got = []
        for n in (1, line, line + 1):
            d = ctx.to_device(k[:n])
            api.op_fft2(ctx, direction, d, d)
            got.append(d.get())
        full = want(k.astype(np.complex128))
        for g in got:
            assert rel_l2(g, full[: len(g)]) < TOL
            assert rel_l2(g, got[-1][: len(g)]) < 4e-7
