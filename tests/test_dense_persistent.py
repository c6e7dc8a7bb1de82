"""The dense solver of small grids in one persistent launch against the split
schedule (which a wait limit below the default selects): grids of one voxel to
either side of the persistent launch's largest, counts that are no multiple of
four, psi that moves voxels out of the band, odd and even iteration counts,
early exits, SDFs with infinite values.  Every voxel of psi and the statistics
must be equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VOXEL = 0.004
KEYS = ("iterations_run", "converged", "diverged", "active_first", "active_last", "max_delta_last")


def both(gpu, shape, P, live, can, psi0, iters):
    nz, ny, nx = shape

    def grid(phi):
        g = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        return g

    gl, gc = grid(live), grid(can)
    out = []
    for limit in (1.0, 0.5):
        prev = gpu.set_wait_limit(limit)
        try:
            f = gpu.Field(gl.dims, gpu.KF_F32)
            f.upload(psi0)
            try:
                st, code = gpu.psi_solve(gl, gc, f, P, iters, "fused"), 0
            except gpu.KFError as e:
                st, code = None, e.status
            out.append((f.download(), st, code))
        finally:
            gpu.set_wait_limit(prev)
    (a, sa, ca), (b, sb, cb) = out
    assert ca == cb
    np.testing.assert_array_equal(a, b)
    if sa is not None:
        for k in KEYS:
            assert sa[k] == sb[k], k
        assert abs(sa["energy_last"] - sb["energy_last"]) <= 1e-12 * abs(sb["energy_last"])
    return a, sa, ca


def random_pair(gpu, shape, P, seed, sigma, fraction=0.2):
    rng = np.random.default_rng(seed)
    live = np.full(shape, P.max_surface + P.epsilon, np.float32)
    can = live.copy()
    pick = rng.random(shape) < fraction
    live[pick] = rng.uniform(-0.9, 0.9, pick.sum()) * P.max_surface
    can[pick] = rng.uniform(-0.9, 0.9, pick.sum()) * P.max_surface
    return live, can, (rng.normal(0.0, 1.0, shape + (3,)) * sigma).astype(np.float32)


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 3, 3), (3, 5, 2), (7, 9, 11), (31, 33, 35), (64, 64, 64),
                                   (98, 98, 98), (107, 107, 108), (107, 108, 108)])
@pytest.mark.parametrize("iters", [1, 2, 5])
@pytest.mark.parametrize("sigma", [0.0, 0.3])
def test_persistent_dense_equals_split(gpu, shape, iters, sigma):
    P = gpu.Params.reference(VOXEL, 5.0)
    live, can, psi0 = random_pair(gpu, shape, P, iters + shape[2], sigma)
    both(gpu, shape, P, live, can, psi0, iters)


@pytest.mark.parametrize("stop", [1, 2, 7])
def test_persistent_dense_early_exit(gpu, stop):
    shape = (21, 22, 23)
    P = gpu.Params.reference(VOXEL, 5.0)
    live, can, psi0 = random_pair(gpu, shape, P, 5, 0.1, 0.05)
    _, st, _ = both(gpu, shape, P, live, can, psi0, stop)
    # the largest step of iteration `stop`: the solve ends there, or sooner
    P = P.with_(early_exit=True, threshold=float(st["max_delta_last"]))
    _, st, _ = both(gpu, shape, P, live, can, psi0, 12)
    assert 1 <= st["iterations_run"] <= stop


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("sigma", [0.0, 0.3])
def test_persistent_dense_non_finite_sdf(gpu, bad, sigma):
    shape = (20, 21, 22)
    P = gpu.Params.reference(VOXEL, 5.0)
    live, can, psi0 = random_pair(gpu, shape, P, 9, sigma)
    live.reshape(-1)[::997] = bad
    both(gpu, shape, P, live, can, psi0, 4)
