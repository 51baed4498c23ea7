"""A grid given with boundary voxels (flag 2) already in it, as a classified
grid exported and set again has them: they stay boundary voxels of material 0
at distance 0, whatever the freed blocks of other rooms held.  Flags, normals,
lists, materials and weights equal the oracle's, for the whole grid and for
slabs."""
import numpy as np
import pytest

import oracle
from virs_b200 import capi, slabs

pytestmark = pytest.mark.gpu


def _use_the_pool(shape, W):
    """Rooms of the same extents whose scratch holds other materials and distances."""
    rng = np.random.default_rng(99)
    n = int(np.prod(shape))
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.02] = 1
    with capi.Simulation(capi.default_params(sponge_width=W)) as s:
        s.set_grid(shape, 0.05, flags, np.full(n, 200, np.uint8))
        s.classify()


def _check(sim, shape, W, flags, wmat):
    want, bm, bd = oracle.classify(shape, W, flags, wmat)
    bidx = oracle.boundary_list(shape, want)
    assert np.array_equal(sim.flags(), want)
    assert np.array_equal(sim.normals(), oracle.normals(shape, want))
    assert np.array_equal(sim.boundary_indices(), bidx)
    m, w = sim.boundary_materials()
    assert np.array_equal(m, bm[bidx])
    assert np.array_equal(w.view(np.uint32), oracle.sponge_weights_for(W, bd[bidx]).view(np.uint32))


@pytest.mark.parametrize("shape,W,density", [((33, 31, 7), 2, 0.05), ((130, 34, 40), 5, 0.001), ((64, 40, 33), 1, 0.0)])
def test_classified_grid_set_again(shape, W, density):
    rng = np.random.default_rng(W)
    n = int(np.prod(shape))
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < density] = 1
    wmat = rng.integers(0, 5, n).astype(np.uint8)
    _use_the_pool(shape, W)
    with capi.Simulation(capi.default_params(sponge_width=W)) as sim:
        sim.set_grid(shape, 0.05, flags, wmat)
        sim.classify()
        given = sim.flags()
        given[rng.random(n) < 0.01] = 2     # ... and some far from any wall, and on the border
        _use_the_pool(shape, W)
        for _ in range(2):
            sim.set_grid(shape, 0.05, given, wmat)
            sim.classify()
            _check(sim, shape, W, given, wmat)
        sim.set_grid(shape, 0.05, flags, wmat)   # without any again
        sim.classify()
        _check(sim, shape, W, flags, wmat)


def test_slabs_of_a_classified_grid():
    shape, W = (40, 33, 30), 2
    rng = np.random.default_rng(3)
    n, plane = int(np.prod(shape)), shape[0] * shape[1]
    flags = np.zeros(n, np.uint8)
    flags[rng.random(n) < 0.02] = 1
    wmat = rng.integers(0, 5, n).astype(np.uint8)
    given, _, _ = oracle.classify(shape, W, flags, wmat)
    want, bm, bd = oracle.classify(shape, W, given, wmat)
    bidx = oracle.boundary_list(shape, want).astype(np.int64)
    _use_the_pool(shape, W)
    got = [], [], []
    for part in range(3):
        with capi.Simulation(capi.default_params(sponge_width=W)) as s:
            slabs.setup_slab(s, shape, 0.05, given, wmat, part, 3, W)
            s.classify()
            z_lo = s.slab_info()[0]
            m, w = s.boundary_materials()
            for g, v in zip(got, (s.boundary_indices().astype(np.int64) + (z_lo - 1) * plane, m, w)):
                g.append(v)
    b, m, w = (np.concatenate(g) for g in got)
    assert np.array_equal(b, bidx)
    assert np.array_equal(m, bm[bidx])
    assert np.array_equal(w.view(np.uint32), oracle.sponge_weights_for(W, bd[bidx]).view(np.uint32))
