"""M and M^T where the contribution lists differ from the smooth mesh's four entries a
target: a mesh that contracts (lists past the eight that sort in registers, and empty
ones), one that expands, an original mesh that is not the identity and one that maps two
entries to a pixel.  The operators keep the reference kernels' rounding and order, so
they equal the oracle's in-order scatter bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import opencliper_gb300 as g
from opencliper_gb300 import api, synth
from oracle import drand48
from oracle import motion as M
from oracle import nesta_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.15, 0.4, 0.8, 1.02])
@pytest.mark.parametrize("mesh", ["identity", "shifted", "doubled"])
@pytest.mark.parametrize("W,H,F", [(40, 32, 1), (64, 48, 3)])
def test_lists(ctx, W, H, F, mesh, scale):
    xn, xm, bb = synth.make_motion(W, H, F, seed=W + F, amplitude=0.3)
    for axis, n in ((0, W), (1, H)):
        c = np.float32(0.5 * (n + 1))
        xn[axis] = c + np.float32(scale) * (xn[axis] - c)
    if mesh == "shifted":
        xm[0] += 1
        xm[1] -= 1
    elif mesh == "doubled":
        xm[0] = (xm[0] // 2) * 2
    rng = np.random.default_rng(int(100 * scale))
    x = (rng.standard_normal((F, H, W)) + 1j * rng.standard_normal((F, H, W))).astype(np.complex64)
    dx, out, dxn, dxm = ctx.to_device(x), ctx.empty(x.shape, np.complex64), ctx.to_device(xn), ctx.to_device(xm)
    api.op_motion(ctx, 1, dx, out, dxn, dxm, bb)
    assert np.array_equal(out.get(), M.warp(x, xn, xm, bb))
    api.op_motion(ctx, 0, dx, out, dxn, dxm, bb)
    assert np.array_equal(out.get(), M.warp_adjoint(x, xn, xm, bb))


@pytest.mark.parametrize("W,H,F", [(40, 32, 2), (64, 48, 5)])
def test_power_method_restart(ctx, W, H, F):
    """The identity as the deformed mesh: U of the constant image is exactly zero, so the
    power method starts over from the drand48 vector (NestaUp.cpp:369-385).  ||U|| and
    the steps against the oracle as in test_motion_gpu.py (2e-3, one step)."""
    p = synth.make_problem(W, H, F, 2, 4, seed=F)
    xn, xm, bb = synth.make_motion(W, H, F, seed=1, amplitude=0.0)
    prob = g.Problem(ctx, ctx.to_device(p.y), ctx.to_device(p.S), ctx.to_device(p.mask))
    prm = dict(lambda_i=0.01, mu_f=1e-3, La=1.0, maxIntIter=1, maxIter=3, stoptest=0, miniter=7, tolVar=3e-4)
    x = ctx.empty((F, H, W), np.complex64)
    prob.run(g.nesta_params(**prm), x)
    x0 = x.get()
    dxn, dxm = ctx.to_device(xn), ctx.to_device(xm)
    prob.set_motion(dxn, dxm, bb)
    s0 = drand48.seed16v_to_state(ctx.rand48())
    st = prob.run(g.nesta_params(**prm), x)
    after = drand48.seed16v_to_state(ctx.rand48())
    prob.close()
    r = R.nesta(p.y, p.S, p.mask, R.NestaParams(**prm), "f32", rand_state=s0, mc=(xn, xm, bb), x_init=x0)
    assert after != s0
    assert abs(st["normU"] - r.stats["normU"]) <= 2e-3 * r.stats["normU"]
    assert abs(st["normest_iters"] - r.stats["normest_iters"]) <= 1
