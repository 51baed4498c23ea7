"""virs_postprocess_ir and virs_postprocess_ir_sinc at the sizes where their
kernels change form: traces shorter than the cascade's lanes are deep, at and
around the staged chunk of 1024 samples, one and 32 sections, more channels
than a warp takes at once, the ends of the window's range."""
import numpy as np
import pytest

import oracle
from virs_b200 import capi

pytestmark = pytest.mark.gpu


def _traces(steps, channels, seed=3):
    rng = np.random.default_rng(seed)
    sim = capi.Simulation(capi.default_params(courant=1.0, boundary_form=1, cell_size=1 / 64))
    n = 20
    flags = np.zeros((n, n, n), np.uint8)
    flags[0] = flags[-1] = flags[:, 0] = flags[:, -1] = flags[:, :, 0] = flags[:, :, -1] = 1
    sim.set_grid((n, n, n), 1 / 64, flags.reshape(-1))
    sim.classify()
    mid = (n // 2 * n + n // 2) * n + n // 2
    sim.set_sources([mid], rng.standard_normal((1, steps)).astype(np.float32))
    sim.set_receivers([mid + k for k in range(-(channels // 2), channels - channels // 2)])
    sim.start(steps)
    sim.run(steps)
    return sim, sim.ir(), float(sim.info().dt)


def _sos(ns, seed=5):
    """Stable sections: pole pairs inside the unit circle, unit gain at rest."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(ns):
        r, th = rng.uniform(0.2, 0.8), rng.uniform(0.1, 2.5)
        a1, a2 = -2 * r * np.cos(th), r * r
        g = (1 + a1 + a2) / 4
        out.append([g, 2 * g, g, 1.0, a1, a2])
    return np.array(out)


@pytest.mark.parametrize("steps,ns", [(3, 1), (3, 32), (61, 32), (62, 32), (63, 2), (1023, 5), (1024, 1), (1025, 32),
                                      (2500, 3)])
def test_cascade_matches_oracle(steps, ns):
    sim, raw, dt = _traces(steps, 3)
    sos = _sos(ns)
    got = sim.postprocess_ir(96000.0, sos, False)
    want = oracle.postprocess(raw, dt, 96000.0, sos, False)
    assert got.shape == want.shape and got.shape[1] > 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    sim.close()


@pytest.mark.parametrize("steps,channels,rate,half,beta,cutoff", [
    (700, 1, 48000.0, 245, 10.06, 0.9167), (700, 8, 16000.0, 64, 8.0, 0.9), (700, 17, 44100.0, 33, 5.0, 0.8),
    (300, 2, 96000.0, 1, 0.0, 1.0), (300, 2, 22050.0, 4096, 50.0, 0.5), (40, 9, 48000.0, 100, 1.0, 0.05)])
def test_sinc_matches_oracle(steps, channels, rate, half, beta, cutoff):
    """FP64 sums of either side: 1e-6 of the peak (both outputs are FP32)."""
    sim, raw, dt = _traces(steps, channels)
    n = int(rate * (steps * dt))
    for normalize in (False, True):
        got = sim.postprocess_ir_sinc(rate, half, beta, cutoff, normalize)
        want = np.stack([oracle.resample_sinc(r, 1.0 / dt, rate, n, half, beta, cutoff, normalize) for r in raw])
        assert got.shape == want.shape and np.abs(want).max() > 0
        assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
    sim.close()
