"""Classification at the sizes where its kernels change form: widths around
the 16 and 32 voxels of a load and a word and the 128 and 512 of a segment
and a warp, rows around a tile's 32, the widest sponge, and rooms whose tiles
are mostly empty.  Flags, normals, lists, materials and weights equal the
oracle's bit for bit."""
import numpy as np
import pytest

import oracle
from virs_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,W,density", [
    ((3, 3, 3), 1, 0.2), ((16, 5, 4), 1, 0.05), ((17, 33, 5), 2, 0.05), ((31, 32, 6), 3, 0.02), ((33, 31, 7), 31, 0.001),
    ((127, 40, 9), 16, 0.0005), ((129, 64, 70), 31, 0.00002), ((513, 34, 5), 8, 0.001), ((640, 70, 12), 1, 0.0),
    ((260, 65, 40), 5, 0.00005)])
def test_classification_matches_oracle(shape, W, density):
    rng = np.random.default_rng(W)
    nx, ny, nz = shape
    flags = np.zeros((nz, ny, nx), np.uint8)
    flags[rng.random(flags.shape) < density] = 1
    flags[rng.random(flags.shape) < density / 4] = 3
    flags[:, :, 0] = 1 # one x wall: the rest of a wide room's tiles see none
    flags = flags.reshape(-1)
    wmat = rng.integers(0, 5, flags.size).astype(np.uint8)
    want, bm, bd = oracle.classify(shape, W, flags, wmat)
    sim = capi.Simulation(capi.default_params(sponge_width=W))
    sim.set_grid(shape, 0.05, flags, wmat)
    for _ in range(2): # again on the same handle: scratch of the first time
        sim.classify()
        bidx = oracle.boundary_list(shape, want)
        assert np.array_equal(sim.flags(), want)
        assert np.array_equal(sim.normals(), oracle.normals(shape, want))
        assert np.array_equal(sim.boundary_indices(), bidx)
        m, w = sim.boundary_materials()
        assert np.array_equal(m, bm[bidx])
        assert np.array_equal(w.view(np.uint32), oracle.sponge_weights_for(W, bd[bidx]).view(np.uint32))
    sim.close()
