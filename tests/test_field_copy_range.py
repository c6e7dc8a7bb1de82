"""kf_field_upload / kf_field_download on a device array whose allocation is
too short: an error, and neighbouring allocations untouched, also where the
array's last byte lies in one of them (here: in another field's planes, which
cudaMalloc places side by side)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["KF_F32", "KF_F64"])
def test_array_past_its_allocation(gpu, precision):
    L = gpu.load()
    dims = (16, 16, 16)
    other, f = (gpu.Field(dims, getattr(gpu, precision)) for _ in range(2))
    rng = np.random.default_rng(3)
    kept = rng.normal(size=other.shape + (3,)).astype(other.dtype)
    mine = rng.normal(size=f.shape + (3,)).astype(f.dtype)
    other.upload(kept)
    f.upload(mine)
    planes = [C.c_void_p() for _ in range(3)]
    gpu.check(L.kf_field_device(other.h, *[C.byref(p) for p in planes]))
    for p in planes:  # each holds a third of the array
        with pytest.raises(gpu.KFError):
            gpu.check(L.kf_field_download(f.h, p, None))
        with pytest.raises(gpu.KFError):
            gpu.check(L.kf_field_upload(f.h, p, None))
    np.testing.assert_array_equal(other.download(), kept)
    np.testing.assert_array_equal(f.download(), mine)
