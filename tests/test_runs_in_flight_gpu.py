"""Calls while a run is in flight on a caller's stream, kept busy for a while
(torch's sleep kernel, about a third of a second) to tell."""
import numpy as np
import pytest

from virs_b200 import capi

pytestmark = pytest.mark.gpu
SLEEP = 600_000_000   # clock cycles


def _room(shape, steps):
    sim = capi.Simulation(capi.default_params(courant=1.0, boundary_form=1))
    flags = np.zeros(shape[::-1], np.uint8)
    flags[:, :, 0] = 1
    sim.set_grid(shape, 0.05, flags.reshape(-1))
    sim.classify()
    mid = ((shape[2] // 2) * shape[1] + shape[1] // 2) * shape[0] + shape[0] // 2
    sim.set_sources([mid], np.random.default_rng(1).standard_normal((1, 40)).astype(np.float32))
    sim.set_receivers([mid, mid + 1])
    sim.start(steps)
    return sim


def test_a_refused_energy_on_the_runs_stream_does_not_hide_it():
    """8193 planes: one more than virs_energy_noalloc takes."""
    import torch
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    sim = _room((5, 5, 8193), 40)
    sim.run(20)
    st = torch.cuda.Stream()
    sim.run(4, st.cuda_stream)
    sim.synchronize()
    with torch.cuda.stream(st):
        torch.cuda._sleep(SLEEP)
    sim.run(4, st.cuda_stream)
    with pytest.raises(capi.VirsError):
        sim.energy_noalloc(out.data_ptr(), st.cuda_stream)
    assert not st.query()
    sim.synchronize()
    assert st.query()
    sim.close()


def test_more_receiver_samples_than_reserved_keep_those_of_a_run_in_flight():
    """1024 are reserved at least; the second run grows them while the first one records."""
    import torch
    shape = (40, 32, 24)
    want = _room(shape, 40)
    want.run(1000)
    want.run(100)
    for second in (None, "the same stream"):
        sim = _room(shape, 40)
        sim.run(4)
        sim.synchronize()
        st = torch.cuda.Stream()
        sim.run(4, st.cuda_stream)
        with torch.cuda.stream(st):
            torch.cuda._sleep(SLEEP)
        sim.run(992, st.cuda_stream)
        sim.run(100, st.cuda_stream if second else None)
        sim.synchronize()
        assert np.array_equal(sim.ir().view(np.uint32), want.ir().view(np.uint32))
        sim.close()
    want.close()
