"""The energy and its gradient on grids that their workspace limit cuts into
parts (9.6 M voxels for the gradient, 67 M for the energy): around the voxel where
the second part begins, against the oracle on the planes around it, with active
voxels there and elsewhere; a value that is not finite in the other part."""
import numpy as np
import pytest

from test_energy_runs import oparams

pytestmark = pytest.mark.gpu

LIMIT = 512 << 20


def long_grid(gpu, nx, ny, nz, seed):
    """A tall grid of a repeated random slab (its repeat no multiple of a part)."""
    P = gpu.Params.reference(0.004, 5.0).with_(gamma_k=0.2)
    rng = np.random.default_rng(seed)
    slab = 37
    tile = lambda a: np.resize(a, (nz,) + a.shape[1:])
    live, can = (tile(rng.uniform(-0.03, 0.03, (slab, ny, nx)).astype(np.float32)) for _ in range(2))
    psi = tile(np.clip(rng.normal(0.0, 0.3, (slab, ny, nx, 3)), -0.9, 0.9).astype(np.float32))
    return P, live, can, psi, rng


def make(gpu, P, live, can, psi):
    dims = live.shape[::-1]
    f = gpu.Field(dims, gpu.KF_F32)
    f.upload(psi)
    grids = []
    for phi in (live, can):
        g = gpu.Grid(dims, 0.004, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, np.ones(phi.shape, np.int32))
        grids.append(g)
    return grids[0], grids[1], f


def f64(*arrays):
    return [a.astype(np.float64) for a in arrays]


@pytest.mark.parametrize("share", [1.0, 0.3])
def test_gradient(gpu, oracle, share):
    nx, ny, nz = 63, 65, 2400
    plane = nx * ny
    part = (LIMIT - 80 * plane) // 56 // 256 * 256
    assert part < nx * ny * nz < 2 * part
    P, live, can, psi, rng = long_grid(gpu, nx, ny, nz, 1)
    gl, gc, f = make(gpu, P, live, can, psi)
    mask = (rng.random(live.shape) < share).astype(np.uint8)
    z = part // plane
    lo, hi = z - 9, z + 9
    got = gpu.energy_adjoint(gl, gc, f, P, mask)
    want = oracle.project_energy_grad(*f64(live[lo:hi], can[lo:hi], psi[lo:hi]), mask[lo:hi], oparams(P))
    inner = slice(5, hi - lo - 5)
    assert np.abs(got[lo:hi][inner] - want[inner]).max() <= 1e-11 * np.abs(want[inner]).max()


def test_gradient_value_not_finite_in_the_other_part(gpu):
    """A voxel of phi_live that is not finite makes 0 times phi_w's derivative not
    finite where a voxel outside the mask samples it, in whichever part."""
    nx, ny, nz = 63, 65, 2400
    P, live, can, psi, _ = long_grid(gpu, nx, ny, nz, 2)
    live[100, 30, 30] = np.inf          # read by its own neighbourhood and, through
    psi[2390, 40, 40] = (-10.0, -10.0, -2290.0)  # psi, by a voxel of the second part
    gl, gc, f = make(gpu, P, live, can, psi)
    mask = np.zeros(live.shape, np.uint8)
    mask[1000:1004, 10:14, 10:14] = 1
    got = gpu.energy_adjoint(gl, gc, f, P, mask)
    assert not np.isfinite(got[2390, 40, 40]).all()
    assert np.isfinite(got[2380:2388]).all() and (got[2380:2388] == 0).all()


def test_energy(gpu, oracle):
    nx, ny, nz = 127, 129, 4224
    plane = nx * ny
    part = (LIMIT - 16 * plane) // 8 // 256 * 256
    assert part < nx * ny * nz < 2 * part
    P, live, can, psi, rng = long_grid(gpu, nx, ny, nz, 3)
    gl, gc, f = make(gpu, P, live, can, psi)
    z = part // plane
    lo, hi = z - 9, z + 9
    mask = np.zeros(live.shape, np.uint8)
    mask[lo + 5:hi - 5] = rng.random((hi - lo - 10, ny, nx)) < 0.5
    got = gpu.energy(gl, gc, f, P, mask).sum()
    want = oracle.project_energy(*f64(live[lo:hi], can[lo:hi], psi[lo:hi]), mask[lo:hi], oparams(P))
    assert abs(got - want) <= 1e-12 * abs(want)
