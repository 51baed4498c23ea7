"""The step in one launch (small grids of default tiling) against the step of
three launches (a tiling set by the caller): the same bits."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu


def _sim(shape, W, seed, storage, sections, n_rcv, rounding=capi.ROUND_NEAREST, tiling=None):
    """Scattered walls and hard sources; soft sources and receivers on every
    kind of voxel, several receivers on one voxel, some on the border."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    n = nx * ny * nz
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.02] = 1
    flags[rng.random(n) < 0.002] = 3
    sim = capi.Simulation(capi.default_params(sponge_width=W, courant=1.0, boundary_form=1, storage=storage))
    sim.set_grid(shape, 0.05, flags, rng.integers(0, 3, n).astype(np.uint8))
    sim.classify()
    one = np.stack([capi.design_octave_cascade(40000.0, a) for a in rng.uniform(0.1, 0.7, (3, 3))])
    coef = np.concatenate([one] * 3, 1)[:, :sections]
    sim.set_filters(coef.astype(np.float32), n_sections=sections)
    x, y, z = np.meshgrid(np.arange(1, nx - 1), np.arange(1, ny - 1), np.arange(1, nz - 1), indexing="ij")
    inner = ((z * ny + y) * nx + x).reshape(-1)
    cls = sim.flags()[inner]
    src = np.concatenate([rng.choice(inner[cls == f], min(2, int((cls == f).sum())), replace=False) for f in range(4)])
    rcv = np.concatenate([src, src[:1], rng.choice(n, n_rcv)])
    steps = 70
    sim.set_sources(src, rng.standard_normal((src.size, steps)).astype(np.float32))
    sim.set_receivers(rcv)
    sim.set_hard_source(rng.standard_normal(20).astype(np.float32))
    sim.set_rounding(rounding)
    if tiling:
        sim.set_tiling(*tiling)
    sim.start(steps)
    for k in (33, 1, 36):
        sim.run(k)
    out = sim.ir(), *sim.pressure(prev=True)
    sim.close()
    return out


@pytest.mark.parametrize("shape,W,storage,sections,n_rcv,rounding", [
    ((32, 32, 5), 1, capi.STORAGE_F32, 1, 4, 0),       # a plane is one block exactly
    ((33, 31, 4), 2, capi.STORAGE_F32, 2, 4, 0),       # ... and a vector less or more
    ((130, 17, 9), 3, capi.STORAGE_F32, 3, 300, 0),    # more probes than threads in a block
    ((5, 4, 3), 1, capi.STORAGE_F32, 4, 4, 0),         # one inner plane
    ((61, 50, 23), 8, capi.STORAGE_F32, 6, 4, 0),      # sections beyond the unrolled ones
    ((61, 50, 23), 8, capi.STORAGE_BF16, 3, 4, 0),
    ((70, 33, 19), 2, capi.STORAGE_F16, 1, 260, 0),
    ((70, 33, 19), 2, capi.STORAGE_F16, 2, 4, 1),
    ((37, 40, 12), 1, capi.STORAGE_BF16, 5, 4, 1),
])
def test_same_bits_as_three_launches(shape, W, storage, sections, n_rcv, rounding):
    a = _sim(shape, W, 7, storage, sections, n_rcv, rounding)
    b = _sim(shape, W, 7, storage, sections, n_rcv, rounding, tiling=(8, 0, 2))
    assert np.abs(a[0]).max() > 0
    for u, v in zip(a, b):
        assert np.array_equal(u.view(np.uint32), v.view(np.uint32))


@pytest.mark.parametrize("storage,sections", [(capi.STORAGE_F32, (3, 3, 3)), (capi.STORAGE_F32, (1, 4, 2)),
                                              (capi.STORAGE_BF16, (2, 6, 1)), (capi.STORAGE_F16, (1, 1, 1))])
def test_small_batch_same_bits_as_three_launches(storage, sections):
    """Members of different sizes, with equal and with different cascades."""
    def members():
        out = []
        for k, (shape, s) in enumerate(zip(((40, 32, 5), (33, 31, 20), (5, 4, 3)), sections)):
            rng = np.random.default_rng(k)
            n = int(np.prod(shape))
            flags = np.zeros(n, np.uint8)
            flags[rng.random(n) < 0.03] = 1
            flags[rng.random(n) < 0.002] = 3
            sim = capi.Simulation(capi.default_params(sponge_width=1 + k, courant=1.0, boundary_form=1, storage=storage))
            sim.set_grid(shape, 0.05, flags, rng.integers(0, 2, n).astype(np.uint8))
            sim.classify()
            coef = np.tile(np.stack([capi.design_octave_cascade(40000.0, a) for a in rng.uniform(0.1, 0.7, (2, 3))]),
                           (1, 2, 1))[:, :s]
            sim.set_filters(coef.astype(np.float32), n_sections=s)
            mid = (shape[2] // 2 * shape[1] + shape[1] // 2) * shape[0] + shape[0] // 2
            sim.set_sources([mid], rng.standard_normal((1, 70)).astype(np.float32))
            sim.set_receivers([mid, mid - 1])
            sim.start(70)
            out.append(sim)
        return out

    got = []
    for tiled in (False, True):
        sims = members()
        b = capi.Batch(sims)
        if tiled:
            b.set_tiling(8, 0, 2)
        for k in (33, 37):
            b.run(k)
        b.synchronize()
        got.append([(s.ir(), *s.pressure(prev=True)) for s in sims])
        b.close()
        for s in sims:
            s.close()
    for x, y in zip(*got):
        assert np.abs(x[0]).max() > 0
        for u, v in zip(x, y):
            assert np.array_equal(u.view(np.uint32), v.view(np.uint32))


@pytest.mark.parametrize("n_rcv", [1, 3])
def test_first_one_launch_step_on_a_callers_stream(n_rcv):
    """The probes of the one-launch step are made inside the run (the timing
    of the parts, on at the start, did not need them) and the run takes
    another stream than the handle's."""
    import torch
    shape, steps = (150, 90, 40), 64
    n = int(np.prod(shape))
    mid = (20 * 90 + 45) * 150 + 75
    out = []
    for late in (False, True):
        sim = capi.Simulation(capi.default_params(sponge_width=1, courant=1.0, boundary_form=1))
        sim.set_grid(shape, 0.05, np.zeros(n, np.uint8), np.zeros(n, np.uint8))
        sim.classify()
        sim.set_sources([mid], np.random.default_rng(3).standard_normal((1, steps)).astype(np.float32))
        sim.set_receivers([mid + k for k in range(n_rcv)])
        sim.set_timing(late)
        sim.start(steps)
        sim.set_timing(False)
        st = torch.cuda.Stream()
        sim.run(steps, st.cuda_stream if late else None)
        sim.synchronize()
        out.append((sim.ir(), *sim.pressure(prev=True)))
        sim.close()
    assert np.abs(out[0][0]).max() > 0
    for u, v in zip(*out):
        assert np.array_equal(u.view(np.uint32), v.view(np.uint32))
