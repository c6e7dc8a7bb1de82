"""The energy's and adjoint's whole-grid passes (runs of 256 voxels, active ones
gathered per CTA, phi_w sampled once) at sizes and masks where the gathering can
go wrong, against the oracle; non-finite psi away from the mask; under capture."""
import numpy as np
import pytest

from oracle.oracle import Params as OParams

pytestmark = pytest.mark.gpu


def oparams(p):
    return OParams(**{k: getattr(p, k) for k in OParams.__dataclass_fields__})


def problem(gpu, dims, seed, precision="KF_F32"):
    P = gpu.Params.reference(0.004, 5.0).with_(gamma_k=0.2)
    shape = dims[::-1]
    rng = np.random.default_rng(seed)
    live, can = (rng.uniform(-0.03, 0.03, shape).astype(np.float32) for _ in range(2))
    f = gpu.Field(dims, getattr(gpu, precision))
    psi = rng.normal(0.0, 0.6, shape + (3,)).astype(f.dtype)
    f.upload(psi)
    grids = []
    for phi in (live, can):
        g = gpu.Grid(dims, 0.004, (0.0, 0.0, 0.0), P.unknown_clip, P)
        g.upload(phi, np.ones(shape, np.int32))
        grids.append(g)
    return P, live, can, psi, grids[0], grids[1], f, rng


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 3, 5), (16, 16, 1), (17, 15, 13), (64, 5, 4), (33, 31, 8)])
@pytest.mark.parametrize("share", [None, 0.0, 0.05, 0.5])
@pytest.mark.parametrize("precision", ["KF_F32", "KF_F64"])
def test_against_oracle(gpu, oracle, dims, share, precision):
    P, live, can, psi, gl, gc, f, rng = problem(gpu, dims, sum(dims), precision)
    mask = np.ones(live.shape, np.uint8) if share is None else (rng.random(live.shape) < share).astype(np.uint8)
    args = (live.astype(np.float64), can.astype(np.float64), psi.astype(np.float64), mask, oparams(P))
    active = None if share is None else mask
    e = gpu.energy(gl, gc, f, P, active).sum()
    want = oracle.project_energy(*args)
    assert abs(e - want) <= 1e-12 * abs(want)
    g = gpu.energy_adjoint(gl, gc, f, P, active)
    og = oracle.project_energy_grad(*args)
    assert np.abs(g - og).max() <= 1e-11 * max(np.abs(og).max(), 1e-300)


def test_non_finite_psi_off_the_mask(gpu):
    """psi that is not finite where no active voxel reads it: 0 times phi_w's
    derivative there, and nothing elsewhere."""
    P, live, can, psi, gl, gc, f, rng = problem(gpu, (24, 20, 16), 5)
    mask = np.zeros(live.shape, np.uint8)
    mask[4:8, 4:8, 4:8] = 1
    clean = gpu.energy_adjoint(gl, gc, f, P, mask)
    psi[12, 12, 12, 0] = np.nan
    f.upload(psi)
    g = gpu.energy_adjoint(gl, gc, f, P, mask)
    assert np.isnan(g[12, 12, 12]).any()
    g[12, 12, 12] = clean[12, 12, 12]
    np.testing.assert_array_equal(g, clean)


def test_adjoint_under_capture(gpu):
    import ctypes as C

    import torch
    P, live, can, psi, gl, gc, f, rng = problem(gpu, (24, 20, 16), 6)
    want = gpu.energy_adjoint(gl, gc, f, P)
    out = torch.zeros(live.shape + (3,), dtype=torch.float64, device="cuda")
    fresh = gpu.Field((24, 20, 16), gpu.KF_F32)
    fresh.upload(psi)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        gpu.check(gpu.load().kf_energy_adjoint(gl.h, gc.h, fresh.h, C.byref(P.c()), None, out.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream))
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
