"""The split schedule's runs without band voxels, tested on phi_live alone where
psi is zero at all of a run's voxels: runs with no, one, some and only moved
voxels beside runs with band voxels, the ragged last run among them.  psi and
the statistics must equal the band-only solver's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VOXEL = 0.004
RUN = 2048


@pytest.mark.parametrize("shape", [(16, 32, 32), (17, 33, 31), (23, 64, 64), (129, 101, 97)])
@pytest.mark.parametrize("moved", ["none", "one", "some", "negative_zero", "all"])
def test_runs_without_band_voxels(gpu, shape, moved):
    nz, ny, nx = shape
    count = nz * ny * nx
    P = gpu.Params.reference(VOXEL, 5.0)
    rng = np.random.default_rng(count)
    live = np.full(count, P.max_surface + P.epsilon, np.float32)
    can = live.copy()
    # band voxels in every third run, psi beside them small; none near the others
    band = np.arange(RUN + 700, count - 600, 3 * RUN)[:, None] + np.arange(0, 300, 7)
    band = band[band < count]
    live[band] = rng.uniform(-0.9, 0.9, band.shape) * P.max_surface
    can[band] = rng.uniform(-0.9, 0.9, band.shape) * P.max_surface
    psi0 = np.zeros((count, 3), np.float32)
    if moved == "one":
        psi0[np.arange(5, count, 2 * RUN), 1] = 0.25
    elif moved == "some":
        psi0[rng.random(count) < 0.01] = 0.3
        psi0[-3:] = -0.2
    elif moved == "negative_zero":
        psi0[:] = -0.0
    elif moved == "all":
        psi0 = rng.normal(0.0, 0.2, psi0.shape).astype(np.float32)
    gl = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
    gc = gpu.Grid((nx, ny, nz), VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
    for g, phi in ((gl, live), (gc, can)):
        phi = phi.reshape(shape)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
    out = []
    prev = gpu.set_wait_limit(1.0)
    try:
        for solver, limit in (("fused", 0.5), ("band", 1.0)):  # (0.5: no persistent dense solver)
            gpu.set_wait_limit(limit)
            f = gpu.Field(gl.dims, gpu.KF_F32)
            f.upload(psi0.reshape(shape + (3,)))
            st = gpu.psi_solve(gl, gc, f, P, 4, solver)
            out.append((f.download(), st))
    finally:
        gpu.set_wait_limit(prev)
    (a, sa), (b, sb) = out
    np.testing.assert_array_equal(a, b)
    assert sa["active_first"] > 0
    for k in ("iterations_run", "active_first", "active_last", "max_delta_last"):
        assert sa[k] == sb[k], k
