"""The float64 solver where each SM has many band voxels (a thread each, in rounds of
equally many warps) and just below: the line at 112 voxels an SM of 152, one
round of 22 warps and one voxel more, shell voxels among them, with and without the
trust-region step, a voxel whose psi is not finite.  psi must equal the oracle's bit
for bit.
"""
import numpy as np
import pytest

from test_group_step import VOXEL, oracle_params, scattered_pair

pytestmark = pytest.mark.gpu


def solve(gpu, live, can, psi0, P, iters):
    grids = []
    for phi in (live, can):
        g = gpu.Grid(phi.shape[::-1], VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        grids.append(g)
    f = gpu.Field(grids[0].dims, gpu.KF_F64)
    f.upload(psi0)
    return f, lambda: gpu.psi_solve(grids[0], grids[1], f, P, iters, "exact")


@pytest.mark.parametrize("count,shell", [(111 * 152, 0), (111 * 152 + 1, 500), (704 * 152, 0), (704 * 152 + 1, 4000)])
@pytest.mark.parametrize("moved,trust", [(False, False), (True, False), (True, True)])
def test_equals_oracle(gpu, oracle, count, shell, moved, trust):
    shape = (33, 41, 39) if count < 20000 else (57, 59, 61)
    P = gpu.Params.reference(VOXEL, 5.0).with_(gamma_k=0.3)
    if trust:
        P = P.with_(use_trust=True, use_killing=False, use_levelset=False)
    live, can = scattered_pair(shape, count, shell, count, P)
    psi0 = np.zeros(shape + (3,))
    if moved:
        psi0 = np.random.default_rng(count).normal(0.0, 0.2, psi0.shape)
    iters = 2
    f, run = solve(gpu, live, can, psi0, P, iters)
    st = run()
    _, want = oracle.solve(live.astype(np.float64), can.astype(np.float64), psi0, iters, oracle_params(P))
    np.testing.assert_array_equal(f.download(), want)
    assert moved or st["active_first"] == count


@pytest.mark.parametrize("count", [3000, 17000])
@pytest.mark.parametrize("data,levelset,killing", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1),
                                                   (0, 0, 0)])
def test_terms_in_use(gpu, oracle, count, data, levelset, killing):
    """The samples of terms that are switched off are not taken."""
    shape = (33, 41, 39)
    P = gpu.Params.reference(VOXEL, 5.0).with_(gamma_k=0.3, use_data=bool(data), use_levelset=bool(levelset),
                                               use_killing=bool(killing))
    live, can = scattered_pair(shape, count, count // 20, count, P)
    psi0 = np.random.default_rng(count).normal(0.0, 0.2, shape + (3,))
    f, run = solve(gpu, live, can, psi0, P, 2)
    run()
    _, want = oracle.solve(live.astype(np.float64), can.astype(np.float64), psi0, 2, oracle_params(P))
    np.testing.assert_array_equal(f.download(), want)


def test_non_finite_psi_stops_the_solve(gpu):
    shape = (33, 41, 39)
    P = gpu.Params.reference(VOXEL, 5.0)
    live, can = scattered_pair(shape, 20000, 0, 3, P)
    psi0 = np.zeros(shape + (3,))
    z, y, x = np.argwhere(np.abs(live) < 0.5 * P.max_surface)[100]
    psi0[z, y, x, 1] = np.nan
    f, run = solve(gpu, live, can, psi0, P, 5)
    with pytest.raises(gpu.DivergedError):
        run()
