"""KF_SOLVER_PERVOXEL's two forms, a warp per voxel where a colour has few voxels and a
thread per voxel where it has many (the line is 9/8 voxel per resident warp, 152 x 16,
half a voxel for one or two steps): the same voxels' psi bit for bit from both (a
band alone, and as part of a larger one that does not touch it), shell voxels and
voxel counts just above and below the line among them.
"""
import numpy as np
import pytest

from test_group_step import VOXEL, scattered_pair

pytestmark = pytest.mark.gpu


def grids(gpu, live, can, P):
    out = []
    for phi in (live, can):
        g = gpu.Grid(phi.shape[::-1], VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        out.append(g)
    return out


@pytest.mark.parametrize("steps", [1, 2, 3, 40])
@pytest.mark.parametrize("more", [5500, 6500, 17000, 18500, 30000])
def test_forms_agree_bit_for_bit(gpu, steps, more):
    shape = (30, 64, 150)
    P = gpu.Params.reference(VOXEL, 5.0)
    few = scattered_pair((30, 64, 70), 4000, 500, 1, P)
    many = scattered_pair((30, 64, 70), more, 2000, 2, P)
    far = np.float32(P.max_surface + P.epsilon)
    psi = []
    for right in (None, many):
        live, can = (np.full(shape, far) for _ in range(2))
        live[:, :, :70], can[:, :, :70] = few
        if right is not None:
            live[:, :, 80:], can[:, :, 80:] = right
        gl, gc = grids(gpu, live, can, P)
        f = gpu.Field(gl.dims, gpu.KF_F32)
        st = gpu.psi_solve(gl, gc, f, P, steps, "pervoxel")
        assert st["active_first"] == 4000 + (more if right is not None else 0)
        psi.append(f.download()[:, :, :70])
    np.testing.assert_array_equal(psi[0], psi[1])
