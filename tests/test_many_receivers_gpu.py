"""More receivers than the one-launch step takes, in one place and all over the
grid: the same bits as the separate kernels, alone and in a batch, and with few
receivers again afterwards."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu
SHAPE, STEPS = (224, 160, 140), 40   # more than 2048 blocks


def _room(rcv, tiling=None):
    nx, ny, nz = SHAPE
    flags = np.zeros(SHAPE[::-1], np.uint8)
    flags[:, :, 0] = flags[:, 0] = flags[0] = 1
    sim = capi.Simulation(capi.default_params(courant=1.0, boundary_form=1))
    sim.set_grid(SHAPE, 0.05, flags.reshape(-1))
    sim.classify()
    mid = (nz // 2 * ny + ny // 2) * nx + nx // 2
    sim.set_sources([mid], np.random.default_rng(2).standard_normal((1, STEPS)).astype(np.float32))
    if tiling:
        sim.set_tiling(*tiling)
    sim.set_receivers(rcv)
    rng = np.random.default_rng(3)
    sim.start(STEPS)
    sim.set_pressure(rng.standard_normal(nx * ny * nz).astype(np.float32))
    return sim


def _out(sim):
    out = sim.ir(), *sim.pressure(prev=True)
    assert np.abs(out[0]).max() > 0
    return out


def _same(a, b):
    assert all(np.array_equal(u.view(np.uint32), v.view(np.uint32)) for u, v in zip(a, b))


@pytest.mark.parametrize("scattered", [False, True])
def test_same_bits_as_the_separate_kernels(scattered):
    n = int(np.prod(SHAPE))
    if scattered:
        rcv = np.random.default_rng(4).choice(n, 9000, replace=False)
    else:
        rcv = SHAPE[0] * SHAPE[1] * 70 + np.arange(9000)
    for r in (rcv, rcv[:4096], rcv[:5]):
        want = _room(r, (8, 0, 2))
        want.run(STEPS)
        got = _room(rcv)
        if r.size < rcv.size:
            got.run(3)
            got.set_receivers(r)
            got.start(STEPS)
            got.set_pressure(np.random.default_rng(3).standard_normal(n).astype(np.float32))
        got.run(33)
        got.run(STEPS - 33)
        _same(_out(got), _out(want))
        got.close()
        sims = [_room(r), _room(rcv[:7])]
        b = capi.Batch(sims)
        b.run(33)
        b.run(STEPS - 33)
        b.synchronize()
        _same(_out(sims[0]), _out(want))
        b.close()
        for s in (want, *sims):
            s.close()
