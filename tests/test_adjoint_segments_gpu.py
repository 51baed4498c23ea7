"""The reverse pass with segments recomputed beside the reverse steps of the
segment after them, against one segment for the whole run: the same signal
gradients bit for bit, the coefficient gradients (FP64 sums in varying order
of fewer than 1e6 terms) to 1e-10."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,sections,tiling", [((40, 33, 20), 2, None), ((5, 4, 3), 1, None),
                                                   ((70, 50, 30), 6, None), ((40, 33, 20), 3, (8, 0, 2))])
def test_segments_do_not_change_the_gradients(shape, sections, tiling):
    rng = np.random.default_rng(5)
    n, steps = int(np.prod(shape)), 23
    sim = capi.Simulation(capi.default_params(sponge_width=1, courant=1.0, boundary_form=1))
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.03] = 1
    mid = (shape[2] // 2 * shape[1] + shape[1] // 2) * shape[0] + shape[0] // 2
    flags[mid:mid + 2] = 0
    sim.set_grid(shape, 0.05, flags, rng.integers(0, 3, n).astype(np.uint8))
    sim.classify()
    coef = np.tile(np.stack([capi.design_octave_cascade(40000.0, a) for a in rng.uniform(0.1, 0.7, (3, 3))]),
                   (1, 2, 1))[:, :sections]
    sim.set_filters(coef.astype(np.float32), n_sections=sections)
    sim.set_sources([mid], rng.standard_normal((1, steps)).astype(np.float32))
    sim.set_receivers([mid, mid + 1])
    if tiling:
        sim.set_tiling(*tiling)
    loss = rng.standard_normal((2, steps)).astype(np.float32)
    got = []
    for every in (steps, 1, 2, 8, 22):
        sim.forward_checkpointed(steps, every)
        got.append(sim.adjoint(loss, 3, sections))
    sim.close()
    (c0, s0), rest = got[0], got[1:]
    assert np.abs(s0).max() > 0
    for c, s in rest:
        assert np.array_equal(s0.view(np.uint32), s.view(np.uint32))
        assert np.allclose(c0, c, rtol=1e-10, atol=1e-10 * np.abs(c0).max())


@pytest.mark.parametrize("sections,form", [(1, 1), (3, 0), (4, 1), (5, 1)])
def test_sources_and_receivers_on_boundary_voxels(sections, form):
    """The receivers' samples are linear in the source signal: the signal
    gradient times the signal is the loss.  Both sums round in single
    precision over 40 steps: 1e-4 of the sum of magnitudes is generous."""
    rng = np.random.default_rng(11)
    shape, steps = (37, 30, 21), 40
    n = int(np.prod(shape))
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.05] = 1
    sim = capi.Simulation(capi.default_params(sponge_width=1, courant=0.5, boundary_form=form))
    sim.set_grid(shape, 0.05, flags, rng.integers(0, 3, n).astype(np.uint8))
    sim.classify()
    bnd = np.flatnonzero(sim.flags().reshape(-1) == 2)
    coef = np.tile(np.stack([capi.design_octave_cascade(40000.0, a) for a in rng.uniform(0.1, 0.7, (3, 3))]),
                   (1, 2, 1))[:, :sections]
    sim.set_filters(coef.astype(np.float32), n_sections=sections)
    sim.set_hard_source(np.zeros(1, np.float32))
    pick = rng.choice(bnd, 40, replace=False)
    sig = rng.standard_normal((10, steps)).astype(np.float32)
    sim.set_sources(pick[:10], sig)
    sim.set_receivers(np.concatenate([pick[5:], pick[5:8]]))  # some on sources, some twice
    loss = rng.standard_normal((38, steps)).astype(np.float32)
    sim.forward_checkpointed(steps, 16)
    terms = loss.astype(np.float64) * sim.ir()[:, :steps]
    _, gs = sim.adjoint(loss, 3, sections)
    sim.close()
    assert np.abs(terms).sum() > 0
    assert abs((gs.astype(np.float64) * sig).sum() - terms.sum()) <= 1e-4 * np.abs(terms).sum()
