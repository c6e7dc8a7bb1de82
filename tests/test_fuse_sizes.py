"""kf_fuse_warped at the grid sizes where the share of a CTA's threads that load
changes (2048 and 8192 voxels per SM of 152), against the oracle bit for bit.  The
smallest form at odd sizes is test_ff_paths.py's."""
import numpy as np
import pytest

from test_ff_paths import oparams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(67, 68, 68), (69, 67, 68), (107, 107, 108), (109, 107, 109)])
@pytest.mark.parametrize("moved", [0.02, 1.0])
def test_either_side_of_a_size(gpu, oracle, dims, moved):
    P = gpu.Params.reference(0.004, 5.0)
    shape = dims[::-1]
    rng = np.random.default_rng(dims[0])
    phi1, phi2 = (rng.uniform(-0.02, 0.02, shape).astype(np.float32) for _ in range(2))
    w1, w2 = (rng.choice([0, 1, 2, 5], shape).astype(np.int32) for _ in range(2))
    psi = (rng.normal(0.0, 0.7, shape + (3,)) * (rng.random(shape + (1,)) < moved)).astype(np.float32)
    f = gpu.Field(dims, gpu.KF_F32)
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
