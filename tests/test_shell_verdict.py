"""The early-exit verdict of the persistent solvers where voxels of the grid's
outer shell alone decide it: a sphere cut by the face z = 0 whose band lies on
the shell only, and one whose interior voxels do not move at all.  The solve must
run to the very iteration whose largest step is the threshold, every time, with
the split schedule's psi (which a wait limit below the default selects).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VOXEL = 0.004
SHAPE = (21, 22, 23)


def cut_sphere_pair(P, interior):
    """Live and canonical SDFs of a sphere on the face z = 0, shifted along x;
    interior "none": unobserved off the shell, "settled": the same in both."""
    nz, ny, nx = SHAPE
    z, y, x = np.mgrid[:nz, :ny, :nx].astype(float)
    far = P.max_surface + P.epsilon

    def sphere(cx):
        d = (np.sqrt((x - cx) ** 2 + (y - ny / 2) ** 2 + z ** 2) - 6.3) * VOXEL
        return np.where(np.abs(d) < P.max_surface, d, far).astype(np.float32)

    can, live = sphere(nx / 2 - 0.4), sphere(nx / 2 + 0.4)
    inner = np.zeros(SHAPE, bool)
    inner[1:-1, 1:-1, 1:-1] = True
    if interior == "none":
        can[inner] = far
    live[inner] = can[inner]
    return live, can


@pytest.mark.parametrize("interior", ["none", "settled"])
@pytest.mark.parametrize("stop", [3, 8, 9])
def test_shell_voxels_keep_the_verdict_open(gpu, interior, stop):
    P = gpu.Params.reference(VOXEL, 5.0)
    if interior == "settled":  # the data term alone: no step where the SDFs agree
        P = P.with_(use_killing=False, use_levelset=False)
    live, can = cut_sphere_pair(P, interior)

    def grid(phi):
        g = gpu.Grid(SHAPE[::-1], VOXEL, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, (phi <= P.max_surface).astype(np.int32))
        return g

    gl, gc = grid(live), grid(can)
    f = gpu.Field(gl.dims, gpu.KF_F32)

    def solve(p, iters, solver, limit):
        prev = gpu.set_wait_limit(limit)
        try:
            f.zero()
            st = gpu.psi_solve(gl, gc, f, p, iters, solver)
            return f.download(), st
        finally:
            gpu.set_wait_limit(prev)

    steps = []
    for k in range(1, stop + 1):
        _, st = solve(P, k, "fused", 0.5)
        steps.append(st["max_delta_last"])
    assert steps[-1] > 0 and all(d > steps[-1] for d in steps[:-1])
    Pe = P.with_(early_exit=True, threshold=float(steps[-1]))
    want, st = solve(Pe, 40, "fused", 0.5)
    assert st["iterations_run"] == stop and st["converged"]
    for _ in range(25):
        for solver in ("fused", "band"):
            got, st = solve(Pe, 40, solver, 1.0)
            assert st["iterations_run"] == stop and st["converged"], solver
            assert st["max_delta_last"] == steps[-1]
            np.testing.assert_array_equal(got, want)
