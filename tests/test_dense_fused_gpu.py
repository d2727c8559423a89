"""The dense passes with the element-wise processes folded in (E, E^H,
SimpleMRIRecon, SimpleMRIReconSOS) where their work splits unevenly, against the
FP64 operators: coil counts around the CTAs of a cluster (1, 2, 3, 5, 9), lengths
with one and several items per thread and with a first factor past 32 (504 = 63 x 8),
partly sampled rows, and a series of several coil groups.  The
per-operator bar of test_ops_gpu.py (1e-5; an FFT of these lengths rounds at
~1e-7)."""
from __future__ import annotations

import numpy as np
import pytest

from opencliper_gb300 import api
from oracle import nesta_ref as R
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _data(W, H, F, C, seed):
    r = np.random.default_rng(seed)
    cx = lambda *s: (r.standard_normal(s) + 1j * r.standard_normal(s)).astype(np.complex64)
    return cx(F, H, W), cx(C, H, W), cx(F, C, H, W), ((r.random((F, H, W)) < 0.6) * 255).astype(np.uint8)


@pytest.mark.parametrize("W,H,F,C", [(8, 8, 1, 1), (24, 40, 2, 2), (512, 24, 1, 3), (40, 504, 1, 5), (200, 280, 2, 9),
                                     (256, 512, 1, 8), (256, 256, 10, 14)])
def test_against_fp64(ctx, W, H, F, C):
    x, S, k, mask = _data(W, H, F, C, W + H + C)
    d = ctx.to_device
    dx, dS, dk, dm = d(x), d(S), d(k), d(mask)
    x64, S64, k64 = x.astype(np.complex128), S.astype(np.complex128), k.astype(np.complex128)
    o = ctx.empty(k.shape, np.complex64)
    api.op_encode(ctx, dx, dS, dm, o)
    got = o.get()
    assert rel_l2(got, R.encode(x64, S64, mask)) < TOL
    assert not got[np.broadcast_to((mask == 0)[:, None], got.shape)].any()
    z = ctx.empty(x.shape, np.complex64)
    for call, want in ((lambda: api.op_encode_adjoint(ctx, dk, dS, z), lambda: R.encode_adjoint(k64, S64)),
                       (lambda: api.simple_recon(ctx, dk, dS, z), lambda: R.simple_recon(k64, S64)),
                       (lambda: api.simple_recon_sos(ctx, dk, z), lambda: R.simple_recon_sos(k64))):
        call()
        assert rel_l2(z.get(), want()) < TOL
    assert np.array_equal(dk.get(), k)
