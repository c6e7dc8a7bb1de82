"""Where float-float and vector paths replaced float64 and scalar ones, bit for
bit against the oracle: integration of 16-bit depth and into voxels that hold
weights, fusion through a displacement field (kept voxels four at a time, moved
ones from a list), and the mesher's test of whole blocks."""
import numpy as np
import pytest

from killingfusion_gb300 import synth
from oracle.oracle import Params as OParams

pytestmark = pytest.mark.gpu


def oparams(p):
    return OParams(**{k: getattr(p, k) for k in OParams.__dataclass_fields__})


@pytest.mark.parametrize("scale", [0.001, 0.0002, 1.0 / 3000.0])
@pytest.mark.parametrize("dims", [(64, 64, 64), (61, 47, 53)])
def test_accumulated_views(gpu, oracle, scale, dims):
    """Five views into one grid, 16-bit and float depth in turn, each view
    against the oracle on the grid's float32 state."""
    grid, frames = synth.sphere_pair()
    P = gpu.Params.paper(grid.voxel)
    v = grid.voxel
    origin = np.array([-0.5 * dims[0] * v, -0.5 * dims[1] * v, 0.4 - 0.5 * dims[2] * v])
    shape = dims[::-1]
    rng = np.random.default_rng(int(1 / scale) + dims[0])
    g = gpu.Grid(dims, v, origin, P.unknown_clip, P)
    phi, w = np.full(shape, np.float32(P.max_surface + P.epsilon)), np.zeros(shape, np.int64)
    for k in range(5):
        c2w = np.eye(4)
        R = synth.rot(rng.normal(size=3) if k else np.array([0.0, 0.0, 1.0]), 0.06 * k)
        c = np.array([0.0, 0.0, 0.4])
        c2w[:3, :3], c2w[:3, 3] = R, c - R @ c
        d = frames[k % 2].astype(np.float64)
        if k % 2 == 0:
            d16 = np.clip(np.rint(d / scale), 0, 65535).astype(np.uint16)
            d16[::37, ::41] = 65535  # values out of range, on both sides
            d16[5::37, 7::41] = 1
            g.integrate_u16(d16, scale, c2w, synth.K, 0.05, 1.2)
            d = d16.astype(np.float64) * scale
        else:
            g.integrate(frames[k % 2], c2w, synth.K, 0.05, 1.2)
        ophi, w = oracle.integrate(phi.astype(np.float64), w, v, origin, P.unknown_clip, d, oracle.invert4(c2w),
                                   synth.K, 0.05, 1.2)
        phi = ophi.astype(np.float32)
        gphi, gw = g.download()
        np.testing.assert_array_equal(gw, w)
        np.testing.assert_array_equal(gphi, phi)
    assert w.max() >= 3


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 1, 1), (2, 3, 1), (17, 13, 11), (32, 32, 32)])
@pytest.mark.parametrize("precision", ["KF_F32", "KF_F64"])
@pytest.mark.parametrize("moved", [0.0, 0.02, 1.0])
def test_fuse_warped(gpu, oracle, dims, precision, moved):
    P = gpu.Params.reference(0.004, 5.0)
    shape = dims[::-1]
    rng = np.random.default_rng(dims[0] * 7 + int(moved * 50))
    phi1, phi2 = (rng.uniform(-0.02, 0.02, shape).astype(np.float32) for _ in range(2))
    w1, w2 = (rng.choice([0, 0, 1, 2, 5, 1 << 24], shape).astype(np.int32) for _ in range(2))
    psi = rng.normal(0.0, 0.7, shape + (3,)) * (rng.random(shape + (1,)) < moved)
    f = gpu.Field(dims, getattr(gpu, precision))
    psi = psi.astype(f.dtype)
    f.upload(psi)
    dst, other = (gpu.Grid(dims, 0.004, (0.0, 0.0, 0.0), P.unknown_clip, P) for _ in range(2))
    dst.upload(phi1, w1)
    other.upload(phi2, w2)
    gpu.fuse_warped(dst, other, f, P)
    gphi, gw = dst.download()
    ophi, ow = oracle.fuse_psi(phi1.astype(np.float64), w1.astype(np.int64), phi2.astype(np.float64),
                               w2.astype(np.int64), psi.astype(np.float64), oparams(P))
    np.testing.assert_array_equal(gw, ow)
    np.testing.assert_array_equal(gphi, ophi.astype(np.float32))


@pytest.mark.parametrize("value", [0.0, "hi", "lo", "nan", "mixed"])
def test_mesh_whole_blocks(gpu, oracle, value):
    """256-cell blocks outside the band but for one cell, wholly above, below,
    above and below, and with a NaN."""
    P = gpu.Params.reference(0.004, 5.0)
    shape = (6, 16, 48)
    hi, lo = np.float32(P.max_surface + P.epsilon), np.float32(-P.unknown_clip - 0.01)
    phi = np.full(shape, hi, np.float32)
    phi[3:] = lo
    if value == "mixed":
        phi.reshape(-1)[::2] = lo
    elif value == "lo":
        phi[:] = lo
    flat = phi.reshape(-1)
    if value in (0.0, "mixed"):
        flat[[0, 255, 256, 700, 1300, flat.size - 1]] = np.float32(-0.003)
    if value == "nan":
        flat[[100, 1500]] = np.nan
    g = gpu.Grid((48, 16, 6), 0.004, (0.0, 0.0, 0.0), P.unknown_clip, P)
    g.upload(phi, np.ones(shape, np.int32))
    tris = gpu.marching_cubes(g, P)
    want = oracle.mesh(phi.astype(np.float64), oparams(P))
    assert len(tris) == len(want)
    if len(want) and value != "nan":
        assert np.abs(tris - want).max() <= 1e-5
