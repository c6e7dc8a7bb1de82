"""The persistent dense solver's test of voxels that have moved (a pass of its own,
a lane per 32nd voxel of its warp's 128) against the split schedule: no such
voxel, single ones, all of them, beside faces (samples partly outside the
grid), at the ends of warps, blocks and the grid.
"""
import numpy as np
import pytest

from test_dense_persistent import both, random_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 8, 4), (5, 5, 5), (16, 32, 33), (61, 63, 65)])
@pytest.mark.parametrize("fraction", [0.0, 1e-4, 0.01, 0.5, 1.0])
@pytest.mark.parametrize("reach", [0.4, 3.0])
def test_moved_voxels(gpu, shape, fraction, reach):
    P = gpu.Params.reference(0.004, 5.0)
    live, can, _ = random_pair(gpu, shape, P, shape[1], 0.0)
    rng = np.random.default_rng(int(fraction * 1e4) + shape[0])
    psi0 = rng.normal(0.0, reach, shape + (3,)).astype(np.float32)
    psi0[rng.random(shape) >= fraction] = 0.0
    flat = psi0.reshape(-1, 3)
    if fraction > 0.0:  # the first and last voxel, and both sides of a warp's and a block's end
        n = len(flat)
        flat[[i for i in (0, 127, 128, 511, 512, n - 1) if i < n]] = (0.3, -0.2, 0.25)
    both(gpu, shape, P, live, can, psi0, 4)
