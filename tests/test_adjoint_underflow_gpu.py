"""Gradients with a loss gradient near the end of FP32's range: the one-launch
reverse step (up to four sections) keeps the subnormals that the separate
kernels of longer cascades keep.  A cascade of two sections and the same one
followed by three sections that pass their input through have the same
gradients: the signal gradients bit for bit, the coefficients' FP64 sums, in
varying order, to 1e-10."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("power", [0, -113, -118])
def test_one_launch_and_separate_kernels_agree(form, power):
    rng = np.random.default_rng(5)
    shape, steps = (36, 30, 24), 80
    n = int(np.prod(shape))
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.03] = 1
    mid = (12 * 30 + 15) * 36 + 18
    flags[mid:mid + 2] = 0
    wmat = rng.integers(0, 3, n).astype(np.uint8)
    two = np.stack([capi.design_octave_cascade(40000.0, a) for a in rng.uniform(0.1, 0.7, (3, 3))])[:, :2]
    five = np.concatenate([two, np.tile(np.array([1.0, 0, 0, 0, 0]), (3, 3, 1))], 1)
    sig = rng.standard_normal((1, steps)).astype(np.float32)
    loss = np.ldexp(rng.standard_normal((2, steps)), power).astype(np.float32)
    got = []
    for coef in (two, five):
        sim = capi.Simulation(capi.default_params(sponge_width=2, courant=0.5, boundary_form=form))
        sim.set_grid(shape, 0.05, flags, wmat)
        sim.classify()
        sim.set_filters(coef.astype(np.float32), n_sections=coef.shape[1])
        sim.set_sources([mid], sig)
        sim.set_receivers([mid + 1, mid + 5])
        sim.set_hard_source(np.zeros(1, np.float32))
        sim.forward_checkpointed(steps, 16)
        gc, gs = sim.adjoint(loss, 3, coef.shape[1])
        got.append((np.array(gc)[:, :2], np.array(gs)))
        sim.close()
    (c2, s2), (c5, s5) = got
    assert np.abs(s2).max() > 0
    assert np.array_equal(s2.view(np.uint32), s5.view(np.uint32))
    assert np.allclose(c2, c5, rtol=1e-10, atol=1e-10 * np.abs(c5).max())
