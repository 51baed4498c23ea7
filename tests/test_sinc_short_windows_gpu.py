"""Sinc resampling around the line between four and 32 lanes per output sample:
window lengths, numbers of output samples that leave groups idle and channel
remainders, against the oracle."""
import numpy as np
import pytest

import oracle
from test_postprocess_shapes_gpu import _traces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half,beta,channels,samples", [
    (1, 0.0, 9, 2500), (2, 50.0, 1, 5000), (3, 8.6, 8, 4999), (32, 8.6, 3, 4503), (33, 8.6, 3, 4503), (32, 8.6, 2, 400),
])
def test_short_windows(half, beta, channels, samples):
    sim, raw, dt = _traces(samples, channels)
    rate, cutoff = 48000.0, 0.83
    n = int(rate * (samples * dt))
    got = sim.postprocess_ir_sinc(rate, half, beta, cutoff, False)
    want = np.stack([oracle.resample_sinc(r, 1.0 / dt, rate, n, half, beta, cutoff, False) for r in raw])
    sim.close()
    assert got.shape == want.shape and np.abs(want).max() > 0
    # FP64 sums of either side, rounded once to FP32
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
