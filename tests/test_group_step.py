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


def oracle_params(P):
    from oracle.oracle import Params
    return Params(**{k: getattr(P, k) for k in Params.__dataclass_fields__})


@pytest.mark.parametrize("count,shell", [(1, 1), (15, 0), (16, 4), (17, 0), (152, 0), (153, 20), (2432, 0), (2433, 80)])
@pytest.mark.parametrize("moved", [False, True])
def test_exact_solver_at_chunk_edges(gpu, oracle, count, shell, moved):
    """The float64 solver's chunks of up to 16 voxels per CTA, bit for bit."""
    shape = (21, 33, 27)
    nz, ny, nx = shape
    P = gpu.Params.reference(VOXEL, 5.0).with_(gamma_k=0.3)
    live, can = scattered_pair(shape, count, shell, 7 * count, P)
    psi0 = np.zeros(shape + (3,))
    if moved:
        psi0 = np.random.default_rng(count).normal(0.0, 0.4, psi0.shape)
    grids = []
    for phi in (live, can):
        g = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        grids.append(g)
    f = gpu.Field((nx, ny, nz), gpu.KF_F64)
    for iters in (1, 4):
        f.upload(psi0)
        gpu.psi_solve(grids[0], grids[1], f, P, iters, "exact")
        _, want = oracle.solve(live.astype(np.float64), can.astype(np.float64), psi0, iters, oracle_params(P))
        np.testing.assert_array_equal(f.download(), want)


@pytest.mark.parametrize("count,shell", [(1, 0), (1, 1), (3, 1), (33, 9), (500, 60), (19500, 0)])
def test_pervoxel_step_at_list_edges(gpu, oracle, count, shell):
    """The per-voxel schedule's colour lists and warps, one step per voxel:
    float32 rounding of one gradient (the bar of one Jacobi iteration)."""
    shape = (25, 33, 27) if count < 19000 else (41, 61, 59)
    nz, ny, nx = shape
    P = gpu.Params.reference(VOXEL, 5.0)
    live, can = scattered_pair(shape, count, shell, 3 * count + 1, P)
    psi0 = np.random.default_rng(count).normal(0.0, 0.05, shape + (3,)).astype(np.float32)
    grids = []
    for phi in (live, can):
        g = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        grids.append(g)
    f = gpu.Field((nx, ny, nz), gpu.KF_F32)
    f.upload(psi0)
    st = gpu.psi_solve(grids[0], grids[1], f, P, 1, "pervoxel")
    r = oracle.solve_pervoxel(live.astype(np.float64), can.astype(np.float64), psi0.astype(np.float64), 1,
                              oracle_params(P), colored=True)
    want = next(v for v in r if isinstance(v, np.ndarray) and v.shape == psi0.shape)
    assert st["active_first"] > 0 or count < 40
    assert np.abs(f.download() - want).max() <= 1e-4


def test_batch_with_shell_voxels_equals_band(gpu):
    """Batched problems with bands off the chunks' 256 voxels and with shell
    voxels (listed apart, a warp each) give their band-only solves' bits."""
    probs, want = [], []
    for k, (shape, count, shell) in enumerate([((9, 11, 13), 40, 40), ((21, 23, 25), 255, 0), ((21, 23, 25), 257, 31),
                                               ((33, 29, 31), 5000, 900), ((5, 4, 3), 60, 54), ((24, 24, 24), 1, 0)]):
        nz, ny, nx = shape
        P = gpu.Params.reference(VOXEL, 5.0).with_(gamma_k=0.2)
        live, can = scattered_pair(shape, count, shell, 40 + k, P)
        psi0 = np.random.default_rng(k).normal(0.0, 0.3, shape + (3,)).astype(np.float32)
        grids = []
        for phi in (live, can):
            g = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
            g.upload(phi, (phi <= P.max_surface).astype(np.int32))
            grids.append(g)
        f = gpu.Field((nx, ny, nz), gpu.KF_F32)
        f.upload(psi0)
        st = gpu.psi_solve(grids[0], grids[1], f, P, 5, "band")
        want.append((f.download(), st["active_first"], st["active_last"], st["max_delta_last"], st["energy_last"]))
        fb = gpu.Field((nx, ny, nz), gpu.KF_F32)
        fb.upload(psi0)
        probs.append((grids[0], grids[1], fb, P))
    batch = gpu.Batch(probs, 5)
    for (_, _, fb, _), w, st in zip(probs, want, batch.run()):
        np.testing.assert_array_equal(fb.download(), w[0])
        assert (st["active_first"], st["active_last"], st["max_delta_last"]) == w[1:4]
        assert abs(st["energy_last"] - w[4]) <= 1e-12 * max(abs(w[4]), 1e-300)
    batch.close()
