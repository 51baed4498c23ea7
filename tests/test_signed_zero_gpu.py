"""The sign of a zero at a boundary voxel: fields at the end of FP32's range,
where the free update flushes to -0 and the centered form divides it by 1 + a.
Equal to the oracle's division bit for bit."""
import numpy as np
import pytest

import oracle
from virs_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiling", [None, (8, 0, 2)])
def test_quotient_keeps_the_sign_of_zero(tiling):
    rng = np.random.default_rng(1)
    shape, W, h = (40, 33, 20), 2, 0.05
    n = int(np.prod(shape))
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.03] = 1
    ref, bm, bd = oracle.classify(shape, W, flags, None)
    bidx = oracle.boundary_list(shape, ref)
    coef = oracle.rbj_highpass_ref(oracle.filter_fs(h, 343.0, 1.0), 440.0, 0.1)[None, None, :]
    air = (ref == 0) | (ref == 2)
    tiny = np.float32(1.3e-38)
    cur = np.where(air & (rng.random(n) < 0.3), rng.choice([-2, -1, 1, 2], n).astype(np.float32) * tiny, np.float32(0.0))
    cur[bidx] = 0.0
    cur = cur.astype(np.float32)
    prev = np.where(air, rng.choice(np.float32([-0.0, 0.0]), n), np.float32(0.0)).astype(np.float32)
    _, c2dt2, inv_h2, K = oracle.step_constants(h, 343.0, 1.0)
    osc = oracle.Scene(shape, ref, bidx, bm[bidx], oracle.sponge_weights_for(W, bd[bidx]), coef, 1,
                       hard=np.zeros(1, np.float32), rcv_idx=bidx[:1].astype(np.uint64), consts=(c2dt2, inv_h2, K), form=1)
    st = (cur.copy(), prev.copy(), np.zeros(bidx.size * 4 + 1, np.float32))
    osc.run(1, state=st)
    zero = st[0][bidx] == 0
    assert (zero & np.signbit(st[0][bidx])).any() and (zero & ~np.signbit(st[0][bidx])).any()
    sim = capi.Simulation(capi.default_params(sponge_width=W, courant=1.0, boundary_form=1))
    sim.set_grid(shape, h, flags)
    sim.classify()
    sim.set_filters(coef.astype(np.float32), n_sections=1)
    sim.set_hard_source(np.zeros(1, np.float32))
    sim.set_receivers(bidx[:1])
    if tiling:
        sim.set_tiling(*tiling)
    sim.start(4)
    sim.set_pressure(cur, prev)
    sim.run(1)
    got = sim.pressure()
    sim.close()
    assert np.array_equal(got[bidx].view(np.uint32), st[0][bidx].view(np.uint32))
