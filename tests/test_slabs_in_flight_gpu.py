"""Slabs that ran on callers' streams, one of them still busy (torch's sleep
kernel, about a third of a second): an exchange and a run of all slabs follow
them, as the handles' completion events do; and a stream in capture, which
cannot wait for such work, is refused."""
import numpy as np
import pytest

from virs_b200 import capi, slabs

pytestmark = pytest.mark.gpu
SLEEP = 600_000_000   # clock cycles
SHAPE, STEPS = (40, 32, 30), 60


def _flags():
    f = np.zeros(SHAPE[::-1], np.uint8)
    f[0] = f[-1] = f[:, 0] = f[:, -1] = f[:, :, 0] = f[:, :, -1] = 1
    return f.reshape(-1)


def _start(sim, p0):
    sim.classify()
    sim.set_hard_source(np.zeros(1, np.float32))
    sim.start(STEPS)
    sim.set_pressure(p0)


def _p0():
    return np.random.default_rng(1).standard_normal(SHAPE[::-1]).astype(np.float32)


def _slabs():
    sims, plane = [], SHAPE[0] * SHAPE[1]
    for r in range(2):
        s = capi.Simulation(capi.default_params())
        lo, hi = slabs.setup_slab(s, SHAPE, 0.05, _flags(), None, r, 2, 1)
        _start(s, _p0().reshape(-1)[(lo - 1) * plane:(hi + 1) * plane])
        sims.append((s, lo, hi))
    return sims


@pytest.mark.parametrize("how", ["exchange", "run", "run of a graph"])
def test_exchange_and_run_follow_what_is_in_flight(how):
    import torch
    whole = capi.Simulation(capi.default_params())
    whole.set_grid(SHAPE, 0.05, _flags())
    _start(whole, _p0())
    steps = 1 if how == "exchange" else 5 if how == "run" else 20
    whole.run(1 + steps)
    want = whole.pressure()
    parts = _slabs()
    sims = [p[0] for p in parts]
    busy = torch.cuda.Stream()
    sims[0].energy_noalloc(torch.zeros(1, dtype=torch.float64, device="cuda").data_ptr(), busy.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(SLEEP)
    capi.slab_exchange(*sims)
    sims[0].run(1, busy.cuda_stream)
    sims[1].run(1)
    if how == "exchange":
        capi.slab_exchange(*sims)
        for s in sims:
            s.run(1)
    else:
        capi.slab_run(sims, steps)
    sims[0].synchronize()
    assert busy.query()
    sims[1].synchronize()
    plane = SHAPE[0] * SHAPE[1]
    for s, lo, hi in parts:
        got = s.pressure().reshape(-1)[plane:(hi - lo + 1) * plane]
        assert np.array_equal(got.view(np.uint32), want.reshape(-1)[lo * plane:hi * plane].view(np.uint32))
    for s in (whole, *sims):
        s.close()


def test_a_stream_in_capture_is_refused():
    import torch
    sim = capi.Simulation(capi.default_params())
    sim.set_grid(SHAPE, 0.05, _flags())
    _start(sim, _p0())
    st = torch.cuda.Stream()
    sim.run(4, st.cuda_stream)
    sim.synchronize()
    graph = torch.cuda.CUDAGraph()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        graph.capture_begin(capture_error_mode="thread_local")
        x += 1
        with pytest.raises(capi.VirsError) as e:
            sim.run(4, st.cuda_stream)
        graph.capture_end()
    assert e.value.status == capi.E_CUDA
    sim.run(4, st.cuda_stream)
    sim.synchronize()
    assert int(sim.info().steps_done) == 8
    sim.close()
