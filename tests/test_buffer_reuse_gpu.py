"""Kept buffers, graphs and freed blocks carry nothing from one use to the
next: every result equals the one of a handle that is used once."""
import threading

import numpy as np
import pytest

from virs_b200 import capi, scenes

pytestmark = pytest.mark.gpu


def _room(n, seed, storage=capi.STORAGE_F32):
    rng = np.random.default_rng(seed)
    nx, ny, nz = n
    flags = np.zeros(nx * ny * nz, np.uint8)
    flags[rng.random(flags.size) < 0.02] = 1
    sim = capi.Simulation(capi.default_params(sponge_width=2, courant=1.0, boundary_form=1, storage=storage))
    sim.set_grid(n, 1 / 64, flags, rng.integers(0, 2, flags.size).astype(np.uint8))
    sim.classify()
    coef = np.stack([capi.design_octave_cascade(40000.0, a)[:2] for a in rng.uniform(0.1, 0.7, (2, 3))])
    sim.set_filters(coef.astype(np.float32), n_sections=2)
    mid = (nz // 2 * ny + ny // 2) * nx + nx // 2
    sim.set_receivers([mid, mid + 1])
    return sim, mid


def _run(sim, mid, steps, seed):
    sig = np.random.default_rng(seed).standard_normal((1, steps)).astype(np.float32)
    sim.set_sources([mid], sig)
    sim.start(steps)
    sim.run(steps)
    return sim.ir().copy(), sim.pressure()


def _same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


@pytest.mark.parametrize("storage", [capi.STORAGE_F32, capi.STORAGE_BF16])
def test_restarts_equal_fresh_handles(storage):
    sim, mid = _room((40, 30, 20), 1, storage)
    for steps, seed in ((70, 1), (70, 2), (33, 3), (2000, 4), (70, 1)):
        got = _run(sim, mid, steps, seed)
        fresh, _ = _room((40, 30, 20), 1, storage)
        assert np.abs(got[0]).max() > 0
        assert _same(got, _run(fresh, mid, steps, seed))
        fresh.close()
    # a restart without new sources, then filters changed in place
    sim.start(70)
    sim.run(70)
    again = sim.ir().copy()
    sim.set_filters(np.zeros((2, 2, 5), np.float32), n_sections=2)
    sim.start(70)
    sim.run(70)
    assert not np.array_equal(again, sim.ir())
    sim.close()


def test_rooms_after_rooms_and_on_two_threads():
    sizes = [(40, 30, 20), (64, 50, 40), (33, 31, 9), (40, 30, 20), (41, 30, 20)]
    want = {}
    for k, n in enumerate(sizes):
        sim, mid = _room(n, k)
        want[k] = _run(sim, mid, 40, k), sim.boundary_indices().copy()
        sim.close()
    bad = []

    def work(order):
        for k in order:
            sim, mid = _room(sizes[k], k)
            if not _same(_run(sim, mid, 40, k), want[k][0]) or not np.array_equal(sim.boundary_indices(), want[k][1]):
                bad.append(k)
            sim.close()

    t = [threading.Thread(target=work, args=(o,)) for o in ([4, 3, 2, 1, 0] * 3, [0, 2, 4, 1, 3] * 3)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not bad


def test_gradients_after_gradients_equal_fresh_handles():
    sc, _ = scenes.inverse_design(steps=80, size=(32, 32, 24), h=0.05)
    kept, _ = scenes.build_simulation(sc)
    for steps, every in ((80, 16), (40, 7), (80, 80), (80, 16)):
        dl = np.random.default_rng(steps + every).standard_normal((4, steps)).astype(np.float32)
        out = []
        for sim in (kept, scenes.build_simulation(sc)[0]):
            sim.forward_checkpointed(steps, every)
            out.append(sim.adjoint(dl, sc.n_materials, sc.n_sections))
            if sim is not kept:
                sim.close()
        # FP64 sums in varying order
        assert np.abs(out[0][0] - out[1][0]).max() <= 1e-10 * np.abs(out[1][0]).max()
        assert np.array_equal(out[0][1], out[1][1])
    kept.close()


def test_step_calls_that_jump_and_mix_with_runs():
    """virs_step uploads its step number only when the counter stands elsewhere."""
    sig = np.random.default_rng(0).standard_normal((1, 64)).astype(np.float32)
    a, mid = _room((40, 30, 20), 1)
    b, _ = _room((40, 30, 20), 1)
    for s in (a, b):
        s.set_sources([mid], sig)
        s.start(64)
    got = [a.step(k)[1] for k in range(5)]
    a.run(3)
    got += [a.step(k)[1] for k in (8, 9)]
    b.run(10)
    want = b.ir()[0]
    assert np.array_equal(np.float32(got[:5]), want[:5]) and np.array_equal(np.float32(got[5:]), want[8:10])
    # a repeated step number reads that step's source sample again
    c, _ = _room((40, 30, 20), 1)
    d, _ = _room((40, 30, 20), 1)
    twice = np.concatenate([sig[:, :4], sig[:, 2:4], sig[:, 40:41]], 1)
    c.set_sources([mid], sig)
    d.set_sources([mid], twice)
    for s in (c, d):
        s.start(64)
    got = [c.step(k)[1] for k in (0, 1, 2, 3, 2, 3, 40)]
    want = [d.step(k)[1] for k in range(7)]
    assert np.array_equal(np.float32(got), np.float32(want))
    for s in (a, b, c, d):
        s.close()
