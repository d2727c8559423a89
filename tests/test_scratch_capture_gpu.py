"""SimpleMRIRecon inside captured CUDA graphs: replays, direct calls and other users of
the context's scratch in every order give the oracle's image.  What a call finds in the
scratch is only what calls that have run left there: a captured call has not run, and a
replay writes the scratch without the host's knowledge.  The scratch is grown first, so
that no call moves it.  The per-operator bar of test_ops_gpu.py."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import opencliper_gb300 as g
from opencliper_gb300 import api
from oracle import nesta_ref as R
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


class _Graph:
    """The launches that `call` makes on the context's stream, captured."""

    def __init__(self, c, call):
        with open("/proc/self/maps") as fh:
            path = sorted({ln.split()[-1] for ln in fh if "libcudart.so" in ln})[0]
        self.rt, self.stream = ctypes.CDLL(path), ctypes.c_void_p(c.stream)
        graph, self.exec = ctypes.c_void_p(), ctypes.c_void_p()
        assert self.rt.cudaStreamBeginCapture(self.stream, 2) == 0  # relaxed
        call()
        assert self.rt.cudaStreamEndCapture(self.stream, ctypes.byref(graph)) == 0
        assert self.rt.cudaGraphInstantiate(ctypes.byref(self.exec), graph, ctypes.c_ulonglong(0)) == 0
        assert self.rt.cudaGraphDestroy(graph) == 0

    def replay(self):
        assert self.rt.cudaGraphLaunch(self.exec, self.stream) == 0

    def close(self):
        assert self.rt.cudaGraphExecDestroy(self.exec) == 0


def test_captured_and_direct_calls_in_any_order(built_lib):
    rng = np.random.default_rng(17)
    cx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    with g.Context(0) as c:
        def shape(W, H, F, C):
            k, S = cx(F, C, H, W), cx(C, H, W)
            dk, dS, x = c.to_device(k), c.to_device(S), c.empty((F, H, W), np.complex64)
            want = R.simple_recon(k.astype(np.complex128), S.astype(np.complex128))
            return (lambda: api.simple_recon(c, dk, dS, x)), x, want, (dk, dS)

        big, _, _, (bk, bS) = shape(96, 80, 3, 5)
        other = lambda: api.op_encode_adjoint(c, bk, bS, c.empty((3, 80, 96), np.complex64))
        a, xa, wa, _ = shape(64, 48, 2, 3)
        b, xb, wb, _ = shape(40, 64, 1, 2)

        def check(call, x, want):
            x.set(np.zeros(x.shape, np.complex64))
            call()
            c.sync()
            got = x.get()
            assert np.isfinite(got).all() and rel_l2(got, want) < TOL

        big()
        check(a, xa, wa)
        check(a, xa, wa)                # a repeated call
        ga = _Graph(c, a)               # captured after one that ran
        other()
        check(ga.replay, xa, wa)        # another user of the scratch in between
        gb = _Graph(c, b)               # a new shape whose first call is captured
        check(b, xb, wb)                # its first direct call, before any replay
        check(gb.replay, xb, wb)
        check(a, xa, wa)
        other()
        gb.replay()                     # a replay between two direct calls of another shape
        check(a, xa, wa)
        gb.replay()
        check(a, xa, wa)
        other()
        check(gb.replay, xb, wb)
        check(ga.replay, xa, wa)
        ga.close()
        gb.close()
