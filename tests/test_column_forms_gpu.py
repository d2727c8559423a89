"""Pixel-mask solves at lengths whose adjoint column pass has two forms, with grids (W/8 x 2
x frames CTAs; 152 SMs) on either side of the lines between them: 420 CTAs run one wave in
both, 480 and 600 one wave in the form without the prefetch alone, 660 two waves in both,
960 two against three.  All rows are kept, more than the pass stages.  The bar of
test_nesta_gpu.py: no further from the FP64 oracle than twice the FP32 restatement."""
from __future__ import annotations

import numpy as np
import pytest

import opencliper_gb300 as g
from opencliper_gb300 import synth
from oracle import drand48
from oracle import nesta_ref as R

pytestmark = pytest.mark.gpu
PRM = dict(lambda_i=0.01, mu_f=1e-3, La=1.0, maxIntIter=1, maxIter=5, stoptest=0, miniter=7, tolVar=3e-4)


@pytest.mark.parametrize("H,F", [(40, 8), (48, 7), (48, 8), (72, 10), (96, 8), (96, 11), (120, 10), (128, 16), (192, 7),
                                 (192, 8), (192, 11)])
def test_pixel_masks(ctx, H, F):
    W, C = 240, 2
    p = synth.make_problem(W, H, F, C, 4, seed=H + F)
    mask = ((np.random.default_rng(H).random((F, H, W)) > 0.6) * 255).astype(np.uint8)
    y = (p.y + 0.05 * synth.make_problem(W, H, F, C, 1, seed=H).y) * (mask != 0)[:, None]
    y = np.ascontiguousarray(y.astype(np.complex64))
    dy, dS, dm, x = ctx.to_device(y), ctx.to_device(p.S), ctx.to_device(mask), ctx.empty((F, H, W), np.complex64)
    prob = g.Problem(ctx, dy, dS, dm)
    rs = drand48.seed16v_to_state(ctx.rand48())  # the power method's restarts draw from it
    stats = prob.run(g.nesta_params(**PRM), x)
    out = x.get()
    prob.close()
    r64 = R.nesta(y, p.S, mask, R.NestaParams(**PRM), "f64", rand_state=rs)
    r32 = R.nesta(y, p.S, mask, R.NestaParams(**PRM), "f32", rand_state=rs)
    assert stats["status"] == 0 and stats["inner_iters"] == PRM["maxIter"]
    assert R.nrmse(out, r64.x) <= 2.0 * R.nrmse(r32.x, r64.x) + 5e-6
