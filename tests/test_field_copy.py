"""kf_field_upload / kf_field_download on device arrays (in place, 16-byte
accesses where the array allows them) against host arrays, at voxel counts off
the 4-voxel vectors and the 1024-voxel blocks, float32 and float64, and from an
array that starts off a 16-byte boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 1, 1), (5, 1, 1), (1023, 1, 1), (32, 32, 1), (41, 25, 1), (33, 31, 29)])
@pytest.mark.parametrize("precision", ["KF_F32", "KF_F64"])
@pytest.mark.parametrize("offset", [0, 1])
def test_device_arrays(gpu, dims, precision, offset):
    import torch
    L = gpu.load()
    prec = getattr(gpu, precision)
    f = gpu.Field(dims, prec)
    n = int(np.prod(dims))
    dt = torch.float32 if precision == "KF_F32" else torch.float64
    want = np.random.default_rng(n).normal(size=f.shape + (3,)).astype(f.dtype)
    f.upload(want)
    flat = torch.full((3 * n + 2,), -7.0, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    gpu.check(L.kf_field_download(f.h, flat[offset:].data_ptr(), None))
    got = flat.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + 3 * n], want.ravel())
    assert np.all(got[:offset] == -7.0) and np.all(got[offset + 3 * n:] == -7.0)
    g = gpu.Field(dims, prec)
    gpu.check(L.kf_field_upload(g.h, flat[offset:].data_ptr(), None))
    np.testing.assert_array_equal(g.download(), want)
