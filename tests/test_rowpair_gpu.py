"""The column-pair row-local iteration (rowpair.cuh) where its work splits
unevenly, against the three-pass iteration on the same data: coil counts
around the four warps of a CTA, the fewest columns and frames, lengths with one,
two and four rounds of second-pass items and with the state in registers and in
tensor memory, rows kept for their data alone, and the recomputed update of the
stopping test.  Both paths round in FP32 only, and 10 iterations do not amplify
that (1e-5, the bound of the every-length test)."""
from __future__ import annotations

import numpy as np
import pytest

import opencliper_gb300 as g
from opencliper_gb300 import synth
from oracle import drand48
from oracle import nesta_ref as R

pytestmark = pytest.mark.gpu

PRM = dict(lambda_i=0.01, mu_f=1e-3, La=1.0, maxIntIter=1, maxIter=10, stoptest=0, miniter=7, tolVar=3e-4)


def _both(ctx, y, S, mask, prm, row_pad=0):
    F, C, H, W = y.shape
    outs, stats = [], []
    for rl in (1, 0):
        ctx.set_tuning("row_local", rl)
        ctx.seed48(drand48.state_to_seed16v(drand48.DEFAULT_STATE))
        try:
            dy, dS, dm = ctx.to_device(y), ctx.to_device(S), ctx.to_device(mask)
            # the image 8 bytes past a 16-byte boundary: callers' images are 8-byte aligned
            buf = ctx.zeros((F * H * W + 2,), np.complex64)
            x = g.DeviceArray(ctx, (F, H, W), np.complex64, ptr=buf.ptr + 8 * row_pad)
            prob = g.Problem(ctx, dy, dS, dm)
            stats.append(prob.run(g.nesta_params(**prm), x))
            outs.append(x.get())
            prob.close()
        finally:
            ctx.set_tuning("row_local", 1)
    return outs, stats


@pytest.mark.parametrize("W,H,F,C", [(8, 32, 2, 1), (8, 256, 2, 2), (24, 128, 3, 3), (16, 192, 3, 4), (40, 72, 2, 5),
                                     (24, 168, 3, 7), (16, 400, 2, 9), (8, 512, 2, 13)])
def test_uneven_splits(ctx, W, H, F, C):
    p = synth.make_problem(W, H, F, C, 8, seed=W + H + C)
    outs, st = _both(ctx, p.y, p.S, p.mask, PRM, row_pad=1)
    assert st[0]["status"] == 0 and st[0]["inner_iters"] == st[1]["inner_iters"] == 10
    assert abs(st[0]["fx_final"] - st[1]["fx_final"]) <= 1e-3 * abs(st[1]["fx_final"])
    assert R.nrmse(outs[0], outs[1]) <= 1e-5


def test_rows_kept_for_their_data(ctx):
    """Nonzero data on rows the mask does not sample, and a frame without any row."""
    p = synth.make_problem(32, 96, 4, 5, 8, seed=3)
    rng = np.random.default_rng(4)
    y, mask = p.y.copy(), p.mask.copy()
    free = [h for h in range(20, 60) if not mask[1, h].any()][:2]
    for h in free:
        y[1, :, h] = (0.05 * (rng.standard_normal((5, 32)) + 1j * rng.standard_normal((5, 32)))).astype(np.complex64)
    y[2], mask[2] = 0, 0
    outs, st = _both(ctx, y, p.S, mask, PRM)
    assert st[0]["kept_rows"] == st[1]["kept_rows"]
    assert R.nrmse(outs[0], outs[1]) <= 1e-5


def test_stopping_test_recomputes_the_last_update(ctx):
    """tolVar so large that the rule fires at the first chance in each of three outer loops."""
    p = synth.make_problem(40, 64, 4, 3, 4, seed=2)
    prm = dict(PRM, maxIntIter=3, maxIter=100, stoptest=1, miniter=4, tolVar=1e30, mu_f=3e-4)
    outs, st = _both(ctx, p.y, p.S, p.mask, prm)
    assert st[0]["inner_iters"] == st[1]["inner_iters"] == 3 * (4 + 2)
    assert R.nrmse(outs[0], outs[1]) <= 1e-5
