"""Receivers on the first and last plane, which no step writes, read a
constant: gradients with and without them are the same (the signal gradients
bit for bit, the coefficient gradients, FP64 sums in varying order, to 1e-10)."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sections", [1, 2, 4, 5])
def test_border_receivers_leave_the_gradients_alone(sections):
    rng = np.random.default_rng(7)
    shape, steps = (24, 20, 16), 60
    nx, ny, nz = shape
    n = int(np.prod(shape))
    flags = np.zeros(n, np.uint8)       # open towards the border
    flags[rng.random(n) < 0.03] = 1
    mid = (nz // 2 * ny + ny // 2) * nx + nx // 2
    flags[mid:mid + 2] = 0
    x, y = rng.integers(2, nx - 2, 12), rng.integers(2, ny - 2, 12)
    border = y * nx + x + np.repeat([0, nz - 1], 6) * nx * ny
    flags[border] = 0
    coef = np.tile(np.stack([capi.design_octave_cascade(40000.0, a) for a in rng.uniform(0.1, 0.7, (3, 3))]),
                   (1, 2, 1))[:, :sections]
    wmat = rng.integers(0, 3, n).astype(np.uint8)
    sig = rng.standard_normal((1, steps)).astype(np.float32)
    loss = rng.standard_normal((1 + border.size, steps)).astype(np.float32)
    got = []
    for rcv in ([mid + 1], [mid + 1, *border]):
        sim = capi.Simulation(capi.default_params(sponge_width=1, courant=0.5, boundary_form=1))
        sim.set_grid(shape, 0.05, flags, wmat)
        sim.classify()
        assert sim.info().boundary_count > 0
        sim.set_filters(coef.astype(np.float32), n_sections=sections)
        sim.set_sources([mid], sig)
        sim.set_receivers(rcv)
        sim.forward_checkpointed(steps, 16)
        got.append(sim.adjoint(loss[:len(rcv)], 3, sections))
        sim.close()
    (c0, s0), (c1, s1) = got
    assert np.abs(s0).max() > 0
    assert np.array_equal(s0.view(np.uint32), s1.view(np.uint32))
    assert np.allclose(c0, c1, rtol=1e-10, atol=1e-10 * np.abs(c0).max())
