"""The sinc window's end: a tap exactly half_taps away is outside, also where
half_taps times its rounded reciprocal is less than one (49, 98, 4087...).
beta 0 keeps the window at one up to the end, and the first output sample has
a tap exactly there."""
import numpy as np
import pytest

import oracle
from test_postprocess_shapes_gpu import _traces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half,beta", [(49, 0.0), (98, 0.0), (103, 2.0), (197, 0.0), (50, 0.0)])
def test_a_tap_at_the_end_is_outside(half, beta):
    sim, raw, dt = _traces(300, 2)
    rate, cutoff = 48000.0, 0.83
    n = int(rate * (300 * dt))
    got = sim.postprocess_ir_sinc(rate, half, beta, cutoff, False)
    want = np.stack([oracle.resample_sinc(r, 1.0 / dt, rate, n, half, beta, cutoff, False) for r in raw])
    sim.close()
    assert np.abs(want).max() > 0
    # FP64 sums of either side, rounded once to FP32
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
