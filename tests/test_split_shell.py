"""The split dense schedule and the trust-region solvers where the band has
voxels on the grid's outer shell, which their band pass deals out to warps by a
list of their positions: none, one, one more and one less than the launch has
warps (16 per SM of 152), all of a small grid's.  psi and the statistics must equal
the band-only solver's bit for bit.
"""
import numpy as np
import pytest

from test_group_step import VOXEL, scattered_pair

pytestmark = pytest.mark.gpu

WARPS = 152 * 16
KEYS = ("iterations_run", "active_first", "active_last", "max_delta_last", "converged", "diverged")


def solve_both(gpu, shape, P, count, shell, iters, moved, limit):
    live, can = scattered_pair(shape, count, shell, count + shell, P)
    grids = []
    for phi in (live, can):
        g = gpu.Grid(shape[::-1], VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        grids.append(g)
    psi0 = np.zeros(shape + (3,), np.float32)
    if moved:
        psi0 = np.random.default_rng(count).normal(0.0, 0.4, psi0.shape).astype(np.float32)
    out = []
    for solver, wait in (("fused", limit), ("band", 1.0)):
        prev = gpu.set_wait_limit(wait)
        try:
            f = gpu.Field(grids[0].dims, gpu.KF_F32)
            f.upload(psi0)
            st = gpu.psi_solve(grids[0], grids[1], f, P, iters, solver)
            out.append((f.download(), st))
        finally:
            gpu.set_wait_limit(prev)
    (a, sa), (b, sb) = out
    np.testing.assert_array_equal(a, b)
    for k in KEYS:
        assert sa[k] == sb[k], k
    assert abs(sa["energy_last"] - sb["energy_last"]) <= 1e-12 * abs(sb["energy_last"])


@pytest.mark.parametrize("count,shell", [(1, 1), (64, 0), (64, 64), (3000, WARPS - 1), (3000, WARPS + 1), (5000, 5000),
                                         (40000, 9000)])
@pytest.mark.parametrize("moved", [False, True])
def test_split_schedule_shell_voxels(gpu, count, shell, moved):
    # large enough for the split schedule by itself
    solve_both(gpu, (107, 109, 111), gpu.Params.reference(VOXEL, 5.0), count, shell, 4, moved, 1.0)


@pytest.mark.parametrize("shape,count,shell", [((3, 3, 3), 27, 26), ((2, 5, 3), 30, 30), ((29, 53, 47), 9000, 4000)])
@pytest.mark.parametrize("moved", [False, True])
def test_split_schedule_small_grids(gpu, shape, count, shell, moved):
    # a wait limit below the default selects the split schedule
    solve_both(gpu, shape, gpu.Params.reference(VOXEL, 5.0), count, shell, 5, moved, 0.5)


@pytest.mark.parametrize("shape,count,shell", [((3, 3, 3), 27, 26), ((29, 53, 47), 500, 60),
                                               ((29, 53, 47), 9000, WARPS + 1)])
@pytest.mark.parametrize("moved", [False, True])
def test_trust_region_shell_voxels(gpu, shape, count, shell, moved):
    P = gpu.Params.reference(VOXEL, 5.0).with_(use_killing=False, use_levelset=False, use_trust=True)
    solve_both(gpu, shape, P, count, shell, 4, moved, 1.0)
