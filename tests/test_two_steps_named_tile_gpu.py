"""Two steps per pass on small grids, with the tile's rows named: left to
itself the library takes single steps there, so these name them and compare
what they are for -- moved sources and the fix list, runs of other lengths
than groups of four, the adjoint's forward pass, batches of members that ran
this way, the reference's own vectors -- with single steps and the oracle, bit
for bit.  And the library's own tile, on a grid large enough that it takes
two steps per pass by itself."""
import numpy as np
import pytest

from test_golden import CASES, RIGID, _load
from test_time_blocking_gpu import _random_case, _same
from virs_b200 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,planes", [(14, 0), (12, 7), (16, 16), (32, 5)])
def test_moved_sources_rebuild_the_fix_list(rows, planes):
    shape, steps = (64, 40, 36), 48
    make, _, _ = _random_case(shape, 1, 21, steps)
    nx, ny, nz = shape
    runs = []
    for pair in (False, True):
        s = make()
        if pair:
            s.set_time_blocking(2, rows, planes)
            assert s.time_blocking()["active"]
        s.run(steps)
        flags = s.flags().reshape(-1)
        k = np.arange(flags.size)
        x, y, z = k % nx, (k // nx) % ny, k // (nx * ny)
        inner = (x > 0) & (y > 0) & (z > 0) & (x < nx - 1) & (y < ny - 1) & (z < nz - 1)
        for at in (0, 2):                           # onto air, then onto boundary voxels
            src = k[inner & (flags == at)]
            s.set_sources(src[[5, len(src) // 2, len(src) - 3]], np.ones((3, 30), np.float32))
            s.start(steps)
            s.run(steps)
            runs.append((s.ir(), *s.pressure(prev=True)))
        s.close()
    for a, b in zip(runs[:2], runs[2:]):
        assert np.abs(a[0]).max() > 0
        assert all(_same(u, v) for u, v in zip(a, b))


@pytest.mark.parametrize("rows,planes", [(14, 0), (16, 5)])
def test_run_lengths_and_single_steps_agree(rows, planes):
    make, want, st = _random_case((70, 45, 33), 2, 11, 55)
    b = make()
    b.set_time_blocking(2, rows, planes)
    for k in (5, 7, 40, 3):
        b.run(k)
    assert _same(b.ir(), want)
    p, pp = b.pressure(prev=True)
    assert _same(p.reshape(-1), st[0]) and _same(pp.reshape(-1), st[1])
    b.close()


def test_adjoint_forward_pass_and_gradients():
    """The forward pass's samples bit for bit; the gradients' FP64 sums, in
    varying order, to 1e-9."""
    sc, _ = scenes.inverse_design(steps=200, size=(40, 36, 28), h=0.04, n_materials=6)
    dl = np.random.default_rng(5).standard_normal((len(sc.rcv_pos), sc.steps)).astype(np.float32)
    out = []
    for pair in (False, True):
        sim, _ = scenes.build_simulation(sc)
        if pair:
            sim.set_time_blocking(2, 14, 16)
        sim.forward_checkpointed(sc.steps, 32)
        out.append((sim.ir(0, sc.steps), *sim.adjoint(dl, sc.n_materials, sc.n_sections)))
        sim.close()
    assert np.abs(out[0][0]).max() > 0 and _same(out[0][0], out[1][0])
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.abs(a - b).max() <= 1e-9 * np.abs(a).max()


def test_batch_of_members_that_ran_two_steps_per_pass():
    shape, steps = (64, 40, 36), 48
    solo, members = [], []
    for seed in (31, 32):
        make, want, _ = _random_case(shape, 1, seed, steps)
        solo.append(want)
        s = make()
        s.set_time_blocking(2, 14, 16)
        s.run(20)                                   # five groups of four
        members.append(s)
    batch = capi.Batch(members)
    batch.run(steps - 20)
    batch.synchronize()
    for m, want in zip(members, solo):
        assert _same(m.ir(), want)
    batch.close()
    for m in members:
        m.close()


@pytest.mark.parametrize("name", CASES + [RIGID])
def test_matches_reference_gpu(name):
    d = _load(name)
    sim = capi.Simulation(capi.default_params(boundary_k=float(d["consts"][3]), rigid_walls=int(name == RIGID)))
    sim.set_grid(tuple(int(s) for s in d["shape"]), float(d["h"]), d["flags_raw"])
    sim.classify()
    sim.set_filters(d["coef"][None, None, :])
    sim.set_receivers(d["rcv"])
    steps = d["ir"].shape[1]
    sim.start(steps)
    sim.set_time_blocking(2, 14, 16)
    sim.run(steps)
    assert _same(sim.ir(), d["ir"])
    assert _same(sim.pressure(), d["p_final"])
    sim.close()


@pytest.mark.parametrize("shape", [(400, 300, 290), (333, 321, 331)])
def test_the_librarys_own_tile(shape):
    """35 M voxels; the spare buffers show that two steps per pass ran."""
    import torch
    rng = np.random.default_rng(4)
    nx, ny, nz = shape
    n, steps = int(np.prod(shape)), 43
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.001] = 1
    mid = (nz // 2 * ny + ny // 2) * nx + nx // 2
    flags[mid - 2:mid + 3] = 0
    sig = rng.standard_normal((2, steps)).astype(np.float32)
    out = []
    for pair in (False, True):
        sim = capi.Simulation(capi.default_params(sponge_width=2, courant=1.0, boundary_form=1))
        sim.set_grid(shape, 0.05, flags)
        sim.classify()
        sim.set_sources([mid, mid + 2], sig)
        sim.set_receivers([mid, mid + 1, mid + 40])
        sim.start(steps)
        if pair:
            sim.set_time_blocking(2)
        capi.trim_memory()
        before = torch.cuda.mem_get_info()[0]
        sim.run(steps)
        sim.synchronize()
        assert (before - torch.cuda.mem_get_info()[0] >= 2 * 4 * n) == pair
        out.append((sim.ir(), *sim.pressure(prev=True)))
        sim.close()
    assert np.abs(out[0][0]).max() > 0
    assert all(_same(u, v) for u, v in zip(*out))
