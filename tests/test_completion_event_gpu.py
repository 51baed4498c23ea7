"""A handle's completion event follows everything queued for it: the next call
takes up after it, and virs_destroy hands its buffers on only then.  A caller's
stream is kept busy for a while (torch's sleep kernel, about a third of a
second) to tell."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu
SLEEP = 600_000_000   # clock cycles


def _room(steps):
    shape = (48, 40, 32)
    sim = capi.Simulation(capi.default_params(courant=1.0, boundary_form=1))
    flags = np.zeros(shape[::-1], np.uint8)
    flags[:, :, 0] = 1
    sim.set_grid(shape, 0.05, flags.reshape(-1))
    sim.classify()
    mid = (16 * 40 + 20) * 48 + 24
    sim.set_sources([mid], np.random.default_rng(1).standard_normal((1, steps)).astype(np.float32))
    sim.set_receivers([mid, mid + 3])
    sim.start(steps)
    return sim


def test_a_refused_call_does_not_hide_a_run_in_flight():
    import torch
    sim = _room(40)
    sim.run(20)
    sim.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        torch.cuda._sleep(SLEEP)
    sim.run(20, st.cuda_stream)
    assert not st.query()
    with pytest.raises(capi.VirsError):      # signals for fewer steps than asked for
        sim.run_host(40, np.zeros((1, 40), np.float32), np.zeros((2, 40), np.float32))
    sim.synchronize()
    assert st.query()
    sim.close()


def test_runs_on_two_streams_and_the_energy_between_are_in_order():
    import torch
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    want = _room(40)
    want.run(20)
    want.energy_noalloc(out[1:].data_ptr(), None)   # its first call loads the kernel, which waits
    want.run(20)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    sim = _room(40)
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(SLEEP)
    sim.run(20, a.cuda_stream)
    sim.energy_noalloc(out.data_ptr(), None)
    sim.run(20, b.cuda_stream)
    assert not a.query()
    sim.synchronize()
    assert a.query() and b.query()
    assert float(out[0]) == float(out[1]) > 0
    assert np.array_equal(sim.ir().view(np.uint32), want.ir().view(np.uint32))
    sim.close()
    want.close()
