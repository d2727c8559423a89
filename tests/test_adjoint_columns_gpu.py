"""The backward columns combined over the coils (k_adj_cols: E^H, SimpleMRIRecon,
SimpleMRIReconSOS) at every column length, whose threads, twiddles and staged tiles
differ by length; with several tiles' coils shared by a cluster and with none; and
with buffers that are 8-byte, not 16-byte aligned.  Against the FP64 operators, the
per-operator bar of test_ops_gpu.py."""
from __future__ import annotations

import numpy as np
import pytest

from opencliper_gb300 import api
from oracle import nesta_ref as R
from tests.conftest import rel_l2
from tests.test_nesta_gpu import LENGTHS

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _check(ctx, W, H, F, C, shift=0):
    r = np.random.default_rng(W + H + C)
    cx = lambda *s: (r.standard_normal(s) + 1j * r.standard_normal(s)).astype(np.complex64)
    k, S = cx(F, C, H, W), cx(C, H, W)
    k64, S64 = k.astype(np.complex128), S.astype(np.complex128)

    def dev(a):  # `shift` values into a buffer of its own
        d = ctx.to_device(np.concatenate([np.zeros(shift, np.complex64), a.ravel()]))
        keep.append(d)
        return api.DeviceArray(ctx, a.shape, np.complex64, ptr=d.ptr + 8 * shift)

    keep = []
    dk, dS, z = dev(k), dev(S), dev(np.zeros((F, H, W), np.complex64))
    for call, want in ((lambda: api.op_encode_adjoint(ctx, dk, dS, z), lambda: R.encode_adjoint(k64, S64)),
                       (lambda: api.simple_recon(ctx, dk, dS, z), lambda: R.simple_recon(k64, S64)),
                       (lambda: api.simple_recon_sos(ctx, dk, z), lambda: R.simple_recon_sos(k64))):
        call()
        assert rel_l2(z.get(), want()) < TOL, (W, H, F, C, shift)


@pytest.mark.parametrize("H", LENGTHS)
def test_every_length(ctx, H):
    _check(ctx, 8, H, 2, 5)      # a cluster's CTAs share the coils unevenly


@pytest.mark.parametrize("W,H,F,C", [(512, 64, 20, 2), (384, 448, 8, 3), (256, 392, 10, 2), (512, 24, 30, 1)])
def test_many_tiles(ctx, W, H, F, C):
    _check(ctx, W, H, F, C)      # a CTA per tile


@pytest.mark.parametrize("W,H,F,C", [(16, 48, 1, 3), (40, 280, 2, 4), (24, 512, 1, 2)])
def test_buffers_aligned_to_one_value(ctx, W, H, F, C):
    _check(ctx, W, H, F, C, shift=1)
