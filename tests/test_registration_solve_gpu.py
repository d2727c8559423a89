"""The one-launch registration descent (k_reg_solve) at the edges of its blocks,
against the restatement: bounding boxes that are no multiple of a tile, control
grids around one block of 8 x 12 points, the fewest frames, a count that is no
multiple of the frames in flight, and one past what the launch takes (which runs
a launch per step).  Bounds as in test_registration_gpu.py: float rounding of
three iterations."""
import numpy as np
import pytest

from opencliper_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,F,radius", [(64, 3, 4), (64, 9, 14), (72, 8, 18), (96, 17, 23), (112, 5, 35), (64, 65, 10)])
def test_descent_matches_restatement(ctx, N, F, radius):
    from oracle import registration as RG
    rng = np.random.default_rng(N + F)
    x = synth.phantom_series(N, N, F, rng)
    x = (x + 0.02 * (rng.standard_normal(x.shape) + 1j * rng.standard_normal(x.shape))).astype(np.complex64)
    kw = dict(radius=radius, nmax=3, W=0.05, lambda_=(0.0, 0.005, 0.0, 0.5))
    ref = RG.Registration(N, F, **kw).run(x)
    r = api.registration(ctx, ctx.to_device(x), api.registration_params(**kw))
    T = r["T"].get()
    assert r["status"] == 0 and r["iterations"] == ref["iterations"]
    assert np.abs(T - ref["T"]).max() <= 1e-5 * np.abs(ref["T"]).max() + 1e-6
    assert np.abs(r["xn"].get() - ref["xn"]).max() <= 5e-5
    np.testing.assert_allclose(r["H"], ref["H"], rtol=1e-5)
