"""The band-only solver's groups of four warps (one lane per voxel, a voxel's
update in parts) at the sizes where their split can go wrong: bands of 1 voxel,
of a lane more or less than a warp's 32 voxels, a group's, a block's and all
blocks' share, voxels on the grid's outer shell (their own path) among them,
and samples that share a corner cell beside samples that do not.  psi and
the statistics must equal the dense solver's bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VOXEL = 0.004


def scattered_pair(shape, count, shell, seed, P):
    """Live and canonical SDFs whose band is `count` random voxels, `shell` of
    them on the outer shell (the rest of the grid unobserved)."""
    rng = np.random.default_rng(seed)
    inner = np.zeros(shape, bool)
    inner[1:-1, 1:-1, 1:-1] = True
    pick = np.concatenate([rng.permutation(np.flatnonzero(~inner))[:shell],
                           rng.permutation(np.flatnonzero(inner))[:count - shell]])
    live = np.full(shape, P.max_surface + P.epsilon, np.float32)
    can = live.copy()
    live.reshape(-1)[pick] = rng.uniform(-0.9, 0.9, len(pick)) * P.max_surface
    can.reshape(-1)[pick] = rng.uniform(-0.9, 0.9, len(pick)) * P.max_surface
    return live, can


@pytest.mark.parametrize("count,shell", [(1, 0), (1, 1), (31, 3), (32, 0), (33, 5), (127, 0), (128, 9), (129, 0),
                                         (4863, 60), (4865, 0), (19456, 0), (19457, 300), (40000, 0)])
@pytest.mark.parametrize("moved", [False, True])
def test_band_equals_dense_at_group_edges(gpu, count, shell, moved):
    shape = (29, 53, 47) if count < 19000 else (41, 61, 59)
    nz, ny, nx = shape
    P = gpu.Params.reference(VOXEL, 5.0)
    live, can = scattered_pair(shape, count, shell, count, P)

    def grid(phi):
        g = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        return g

    gl, gc = grid(live), grid(can)
    psi0 = np.zeros(shape + (3,), np.float32)
    if moved:
        psi0 = np.random.default_rng(count + 1).normal(0.0, 0.4, psi0.shape).astype(np.float32)
    out = []
    for solver in ("fused", "band"):
        f = gpu.Field(gl.dims, gpu.KF_F32)
        f.upload(psi0)
        st = gpu.psi_solve(gl, gc, f, P, 3, solver)
        out.append((f.download(), st["active_first"], st["active_last"], st["max_delta_last"], st["energy_last"]))
    a, b = out
    if not moved:
        assert a[1] == count
    np.testing.assert_array_equal(a[0], b[0])
    assert a[1:4] == b[1:4]
    assert abs(a[4] - b[4]) <= 1e-12 * abs(a[4])
