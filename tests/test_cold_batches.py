"""The split schedule's runs without band voxels where a block tests several of them
at once (all with zero psi) and where some of its runs have moved voxels: band
voxels in few runs, at the first and the last run or at neither, voxel counts off
four and off a run.  psi and the statistics must equal the band-only solver's.
"""
import numpy as np
import pytest

from test_cold_runs import RUN, VOXEL
from test_split_shell import KEYS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(17, 33, 31), (41, 47, 43), (109, 108, 107)])
@pytest.mark.parametrize("where", [0, 3, -1])
@pytest.mark.parametrize("moved", [0, 1, 7, 10**9])
def test_few_hot_runs(gpu, shape, where, moved):
    nz, ny, nx = shape
    count = nz * ny * nx
    runs = count // 4 // (RUN // 4)
    P = gpu.Params.reference(VOXEL, 5.0)
    rng = np.random.default_rng(count)
    live = np.full(count, P.max_surface + P.epsilon, np.float32)
    can = live.copy()
    band = (where % max(runs, 1)) * RUN + 900 + np.arange(0, 300, 7)
    live[band] = rng.uniform(-0.9, 0.9, band.shape) * P.max_surface
    can[band] = rng.uniform(-0.9, 0.9, band.shape) * P.max_surface
    psi0 = np.zeros((count, 3), np.float32)
    if moved:  # every moved-th run has a moved voxel
        psi0[np.arange(min(moved, 2) * RUN + 5, count, moved * RUN), 1] = 0.25
    grids = []
    for phi in (live, can):
        g = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi.reshape(shape), (phi.reshape(shape) <= P.max_surface).astype(np.int32))
        grids.append(g)
    out = []
    for solver, limit in (("fused", 0.5), ("band", 1.0)):
        prev = gpu.set_wait_limit(limit)
        try:
            f = gpu.Field(grids[0].dims, gpu.KF_F32)
            f.upload(psi0.reshape(shape + (3,)))
            st = gpu.psi_solve(grids[0], grids[1], f, P, 4, solver)
            out.append((f.download(), st))
        finally:
            gpu.set_wait_limit(prev)
    (a, sa), (b, sb) = out
    np.testing.assert_array_equal(a, b)
    assert sa["active_first"] > 0
    for k in KEYS:
        assert sa[k] == sb[k], k
