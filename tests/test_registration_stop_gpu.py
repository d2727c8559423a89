"""The one-launch registration descent ended by its stopping rule: |Dif| falls below the
threshold at iterations 7 and 8 (the metric's own threshold is always met), so the
iterations done, and the buffer T ends in, come from the partial sums of |Dif|^2.
|Dif| of the iterations around the threshold lies 4 % or more from it.  Bounds: those of test_registration_solve_gpu.py for
three iterations, times the iterations here (8 / 3)."""
import numpy as np
import pytest

from opencliper_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("et,last", [(0.0942, 7), (0.0858, 8)])
def test_stopped_by_the_step_size(ctx, et, last):
    from oracle import registration as RG
    N, F = 64, 6
    rng = np.random.default_rng(N + F)
    x = synth.phantom_series(N, N, F, rng)
    x = (x + 0.02 * (rng.standard_normal(x.shape) + 1j * rng.standard_normal(x.shape))).astype(np.complex64)
    kw = dict(radius=12, nmax=30, W=0.05, lambda_=(0.0, 0.005, 0.0, 0.5), et=et, eh=0.5)
    ref = RG.Registration(N, F, **kw).run(x)
    assert ref["iterations"] == last
    r = api.registration(ctx, ctx.to_device(x), api.registration_params(**kw))
    assert r["status"] == 0 and r["iterations"] == last
    T = r["T"].get()
    assert np.abs(T - ref["T"]).max() <= 3e-5 * np.abs(ref["T"]).max() + 3e-6
    np.testing.assert_allclose(r["H"], ref["H"], rtol=3e-5)
