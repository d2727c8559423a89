"""The element-wise processes, which take pairs of values, against the FP64 operators:
on 16-byte aligned buffers and on buffers one value off (the results must be the same
bits), one row and one frame, more frames or coils than a grid dimension holds, an odd
count for the normalisation.  FP32 with at most nine terms a sum: 1e-6."""
from __future__ import annotations

import numpy as np
import pytest

from opencliper_gb300 import api
from opencliper_gb300.api import DeviceArray
from oracle import nesta_ref as R
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _put(ctx, a, off, keep):
    """`a` on the device, `off` elements past an allocation's start."""
    base = ctx.empty((a.size + off,), a.dtype)
    keep.append(base)
    v = DeviceArray(ctx, a.shape, a.dtype, ptr=base.ptr + off * a.itemsize)
    return v.set(a)


def _run(ctx, x, S, k, mask, off):
    keep, out = [], {}
    put = lambda a: _put(ctx, a, off, keep)
    dx, dS, dk, dm = put(x), put(S), put(k), put(mask)
    new = lambda a: put(np.zeros_like(a))
    for name, like, call in (("fwd", x, lambda o: api.op_ttv(ctx, 1, dx, o)), ("bwd", x, lambda o: api.op_ttv(ctx, 0, dx, o)),
                             ("norm", x, lambda o: api.op_normalize(ctx, dx, o, 0.5)),
                             ("prod", k, lambda o: api.op_sensmul(ctx, False, dx, dS, o)),
                             ("conj", k, lambda o: api.op_sensmul(ctx, True, dk, dS, o)),
                             ("sum", x, lambda o: api.op_coilsum(ctx, dk, o)), ("rss", x, lambda o: api.op_rss(ctx, dk, o))):
        o = new(like)
        call(o)
        out[name] = o.get()
    api.op_mask(ctx, dk, dm)
    out["mask"] = dk.get()
    return out


@pytest.mark.parametrize("W,H,F,C", [(8, 1, 1, 1), (24, 5, 1, 3), (56, 9, 4, 9), (512, 40, 3, 2), (8, 1, 65540, 1),
                                     (8, 1, 1, 65540)])
def test_pairs(ctx, W, H, F, C):
    r = np.random.default_rng(W + H + F + C)
    cx = lambda *s: (r.standard_normal(s) + 1j * r.standard_normal(s)).astype(np.complex64)
    x, S, k = cx(F, H, W), cx(C, H, W), cx(F, C, H, W)
    mask = ((r.random((F, H, W)) < 0.5) * 255).astype(np.uint8)
    got = _run(ctx, x, S, k, mask, 0)
    x64, S64, k64 = x.astype(np.complex128), S.astype(np.complex128), k.astype(np.complex128)
    assert np.array_equal(got["mask"], R.apply_mask(k, mask))
    want = {"fwd": R.ttv(x64, True), "bwd": R.ttv(x64, False), "norm": R.normalize(x64, 0.5),
            "prod": R.sensmul(x64, S64, False), "conj": R.sensmul(k64, S64, True), "rss": R.rss(k64)}
    if C <= 9:  # a longer sum rounds more
        want["sum"] = R.coilsum(k64)
    else:
        del want["rss"]
    for name, w in want.items():
        err = rel_l2(got[name], w) if np.any(w) else float(np.abs(got[name]).max())
        assert err < TOL, (name, err)
    off = _run(ctx, x, S, k, mask, 1)
    for name in got:
        assert np.array_equal(got[name], off[name]), name


@pytest.mark.parametrize("n", [1, 2, 7, 513])
def test_normalize_odd_counts(ctx, n):
    r = np.random.default_rng(n)
    x = (r.standard_normal(n + 1) + 1j * r.standard_normal(n + 1)).astype(np.complex64)
    d, o = ctx.to_device(x), ctx.to_device(np.zeros_like(x))
    a, b = DeviceArray(ctx, (n,), np.complex64, ptr=d.ptr), DeviceArray(ctx, (n,), np.complex64, ptr=o.ptr)
    api.op_normalize(ctx, a, b, 0.7)
    got = o.get()
    assert got[n] == 0 and rel_l2(got[:n], R.normalize(x[:n].astype(np.complex128), 0.7)) < TOL
