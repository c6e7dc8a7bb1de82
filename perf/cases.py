"""The performance cases of the registration loop: what a program that uses the
library calls, at the sizes, types and options of the project's workloads.

Kinds of case
  solve      one displacement solve from a zero field (kf_field_zero,
             kf_psi_solve, psi read back to the device as [N][3]);
  batch      many uneven problems solved together (kf_batch_run);
  integrate  one SDF from several posed depth views (kf_compute_sdf for the
             first, kf_integrate_depth for the others);
  mesh       an SDF fused through a displacement field into a new SDF and
             meshed (kf_grid_reset, kf_fuse_warped, kf_marching_cubes_async);
  energy     the differentiable energy and its gradient (kf_energy,
             kf_energy_adjoint);
  sequence   a first frame and the frames after it through FramePipeline:
             integration, solve, warp + fuse and three meshes per frame.
"""
import ctypes as C
import math

import numpy as np
import torch

from killingfusion_gb300 import capi, pipeline, synth

DEV = "cuda"
ORIGIN = (-0.64, -0.64, 0.30)  # the ellipsoid scene's box: 1.28 m a side


def listed():
    return [
        # the smallest registration: the 64^3 sphere pair with the default
        # solver; launches and latencies, everything in L2
        {"name": "solve_dense_64", "kind": "solve", "scene": "sphere", "solver": "fused",
         "nx": 64, "ny": 64, "nz": 64, "iterations": 100},
        # the headline: every voxel tested in each of 200 iterations at 256^3
        {"name": "solve_dense_256", "kind": "solve", "scene": "ellipsoids", "solver": "fused",
         "nx": 256, "ny": 256, "nz": 256, "iterations": 200},
        # the same registration with the solver a live system would use
        {"name": "solve_band_256", "kind": "solve", "scene": "ellipsoids", "solver": "band",
         "nx": 256, "ny": 256, "nz": 256, "iterations": 200},
        # the reference's default schedule (each voxel to convergence), on a
        # grid cut to the object's box
        {"name": "solve_pervoxel_117", "kind": "solve", "scene": "ellipsoids", "solver": "pervoxel",
         "nx": 117, "ny": 101, "nz": 93, "iterations": 100},
        # the float64 replay that a result is checked against
        {"name": "solve_exact_64", "kind": "solve", "scene": "sphere", "solver": "exact",
         "nx": 64, "ny": 64, "nz": 64, "iterations": 20},
        # offline registration of a whole collection
        {"name": "batch_64", "kind": "batch", "problems": 64, "lo": 34, "hi": 156, "iterations": 150},
        # an SDF accumulated from four views of a moving 16-bit depth camera
        {"name": "integrate_u16_250", "kind": "integrate", "u16": True, "views": 4,
         "nx": 250, "ny": 231, "nz": 243},
        # the registered mesh of a frame (SDF::getMesh through psi)
        {"name": "mesh_warped_251", "kind": "mesh", "nx": 251, "ny": 256, "nz": 233},
        # energy and gradient for an outer optimiser
        {"name": "energy_128", "kind": "energy", "nx": 121, "ny": 128, "nz": 115},
        # a small interactive loop, bound by launches and the host
        {"name": "sequence_band_64", "kind": "sequence", "scene": "sphere", "solver": "band",
         "n": 64, "frames": 3, "iterations": 100},
        # the live system at the headline size
        {"name": "sequence_band_256", "kind": "sequence", "scene": "ellipsoids", "solver": "band",
         "n": 256, "frames": 4, "iterations": 200},
        # the large grid with the default solver, 300 iterations a frame
        {"name": "sequence_dense_512", "kind": "sequence", "scene": "capsules", "solver": "fused",
         "n": 512, "frames": 2, "iterations": 300},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """A box of about an n^3 grid's size, odd sides among them."""
    n = _log(rng, lo, hi)
    side = lambda: max(lo, min(hi, n + rng.randint(-n // 10, n // 10)))  # noqa: E731
    return {"nx": side(), "ny": side(), "nz": side()}


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "integrate", "mesh", "energy", "sequence"])
    if kind == "solve":
        solver = rng.choice(["fused", "band", "band", "pervoxel", "exact"])
        hi = {"fused": 288, "band": 400, "pervoxel": 192, "exact": 96}[solver]
        its = {"fused": (50, 250), "band": (50, 300), "pervoxel": (50, 100), "exact": (10, 30)}[solver]
        return {"kind": kind, "scene": "ellipsoids", "solver": solver, **_box(rng, 48, hi),
                "iterations": rng.randint(*its)}
    if kind == "batch":
        lo = _log(rng, 16, 48)
        return {"kind": kind, "problems": _log(rng, 4, 96), "lo": lo, "hi": lo + _log(rng, 16, 90),
                "iterations": rng.randint(50, 150)}
    if kind == "integrate":
        return {"kind": kind, "u16": rng.random() < 0.5, "views": rng.randint(1, 5), **_box(rng, 64, 384)}
    if kind == "mesh":
        return {"kind": kind, **_box(rng, 64, 384)}
    if kind == "energy":
        return {"kind": kind, **_box(rng, 32, 160)}
    return {"kind": kind, "scene": "ellipsoids", "solver": rng.choice(["fused", "band", "band"]),
            "n": _log(rng, 64, 288), "frames": rng.randint(2, 4), "iterations": rng.randint(50, 200)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _sequence(scene, n, seed):
    if scene == "sphere":
        return synth.SpherePairSequence(seed=1 + seed)
    if scene == "capsules":
        return synth.CapsuleSequence(seed=5 + seed, n=n)
    return synth.EllipsoidSequence(seed=2 + seed, n=n)


def _placement(case):
    """Voxel size and min corner of a solve or mesh case's grid: the scene's
    own for the sphere pair; for the ellipsoids the voxel that lets the
    longest side cover the scene's box, the grid centred in it."""
    if case.get("scene") == "sphere":
        v = 0.004
        return v, np.array([-32 * v, -32 * v, 0.4 - 32 * v])
    dims = _dims(case)
    v = 1.28 / max(dims)
    return v, np.array([ORIGIN[k] + 0.5 * (1.28 - dims[k] * v) for k in range(3)])


def _params(voxel, trunc=5.0):
    return capi.Params.reference(voxel, trunc)


def _tsdf(phi, w, depth, c2w, dims, voxel, origin, clip, lo=0.05, hi=1.2):
    """SDF::integrateDepthFrame in float64: phi, w (flat, float64) after one
    more depth view (float64 [h, w])."""
    nx, ny, nz = dims
    W = np.linalg.inv(np.asarray(c2w, dtype=np.float64))
    K = synth.K
    ax = lambda n, k: voxel * (torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) + float(origin[k])  # noqa: E731
    X, Y, Z = ax(nx, 0).view(1, 1, nx), ax(ny, 1).view(1, ny, 1), ax(nz, 2).view(nz, 1, 1)
    c = [((W[r, 0] * X + W[r, 1] * Y) + W[r, 2] * Z) + W[r, 3] for r in range(3)]
    a, b = c[0] / c[2], c[1] / c[2]
    u = (K[0, 0] * a + K[0, 1] * b) + K[0, 2]
    v = (K[1, 0] * a + K[1, 1] * b) + K[1, 2]
    del a, b

    def pixel(t):  # roundf of the float32 value, halves away from zero
        f = (t + 0.5).to(torch.float32).to(torch.float64)
        return torch.where(torch.isfinite(f), torch.sign(f) * torch.floor(f.abs() + 0.5), torch.full_like(f, -1.0))

    col, row = pixel(u), pixel(v)
    h, wd = depth.shape
    ok = (col >= 0) & (col < wd) & (row >= 0) & (row < h)
    k = (torch.where(ok, row, 0.0) * wd + torch.where(ok, col, 0.0)).to(torch.int64)
    d = depth.reshape(-1)[k]
    dist = d - c[2].expand_as(d)
    ok &= (d >= lo) & (d <= hi) & (dist >= -clip)
    ok, dist = ok.reshape(-1), dist.reshape(-1)
    return torch.where(ok, (phi * w + dist) / (w + 1.0), phi), torch.where(ok, w + 1.0, w)


def _scene_sdfs(case, seed):
    """float32 (live, canonical) SDFs of two depth frames with the weights of
    the live one, flat on the device, and the parameters and placement."""
    voxel, origin = _placement(case)
    dims = _dims(case)
    P = _params(voxel)
    seq = _sequence(case.get("scene", "ellipsoids"), 256, seed)
    out = []
    for f in (1, 0):
        d = torch.from_numpy(seq.frame(f)).to(DEV).double()
        n = dims[0] * dims[1] * dims[2]
        phi = torch.full((n,), P.max_surface + P.epsilon, dtype=torch.float64, device=DEV)
        phi, w = _tsdf(phi, torch.zeros_like(phi), d, np.eye(4), dims, voxel, origin, P.unknown_clip)
        out += [phi.float(), w.to(torch.int32)]
    return out[0], out[2], out[1], out[3], P, voxel, origin


def _smooth_psi(dims, rng, amp):
    """A smooth displacement field [nz, ny, nx, 3], float64: 8 Gaussians."""
    nx, ny, nz = dims
    x, y, z = (torch.arange(n, dtype=torch.float64, device=DEV) for n in dims)
    psi = torch.zeros((nz, ny, nx, 3), dtype=torch.float64, device=DEV)
    for _ in range(8):
        c = rng.uniform(0.2, 0.8, 3) * np.array(dims)
        s = rng.uniform(0.06, 0.2) * max(dims)
        g = lambda t, k: torch.exp(-((t - c[k]) ** 2) / (2 * s * s))  # noqa: E731
        e = g(z, 2).view(nz, 1, 1) * g(y, 1).view(1, ny, 1) * g(x, 0).view(1, 1, nx)
        psi += e[..., None] * torch.tensor(rng.uniform(-amp, amp, 3), device=DEV)
    return psi * min(1.0, amp / float(psi.abs().max()))


def _shape_sdfs(n, rng):
    """A sphere, ellipsoid or torus filling about half of an n^3 grid and the
    same shape offset by up to 3 voxels and bent: (canonical, live), voxel."""
    kind = int(rng.integers(0, 3))
    size = 0.10
    voxel = 2.0 * size / n
    t = (torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * voxel - n * voxel / 2
    X, Y, Z = t.view(1, 1, n), t.view(1, n, 1), t.view(n, 1, 1)
    off = rng.uniform(-3.0, 3.0, 3) * voxel
    bend = rng.uniform(-0.15, 0.15)
    a = rng.uniform(0.6, 1.0, 3) * size * 0.45
    trunc = 5.0 * voxel

    def sdf(X, Y, Z):
        if kind == 0:
            d = torch.sqrt(X * X + Y * Y + Z * Z) - a[0]
        elif kind == 1:
            d = (torch.sqrt((X / a[0]) ** 2 + (Y / a[1]) ** 2 + (Z / a[2]) ** 2) - 1.0) * a.min()
        else:
            q = torch.sqrt(X * X + Z * Z) - a[0]
            d = torch.sqrt(q * q + Y * Y) - a[0] * 0.35
        return torch.where(d > trunc, trunc + 1e-5, d.clamp(min=-trunc - 1e-3)).float().reshape(-1)

    Xl = X - off[0]
    return sdf(X, Y, Z), sdf(Xl, Y - off[1] - bend * (Xl / size) ** 2 * size, Z - off[2]), voxel


def _blobs(dims, rng, voxel):
    """Truncated SDF of 16 random Gaussian blobs, float32 flat."""
    nx, ny, nz = dims
    n = max(dims)
    X, Y, Z = ((torch.arange(m, dtype=torch.float64, device=DEV) + 0.5) * voxel for m in dims)
    X, Y, Z = X.view(1, 1, nx), Y.view(1, ny, 1), Z.view(nz, 1, 1)
    f = torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
    g = [torch.zeros_like(f) for _ in range(3)]
    for _ in range(16):
        c = rng.uniform(0.25, 0.75, 3) * np.array(dims) * voxel
        s = rng.uniform(0.02, 0.08) * n * voxel
        d = (X - c[0], Y - c[1], Z - c[2])
        e = rng.uniform(0.5, 1.0) * torch.exp(-(d[0] ** 2 + d[1] ** 2 + d[2] ** 2) / (2 * s * s))
        f += e
        for k in range(3):
            g[k] -= e * d[k] / (s * s)
    gn = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2) + 1e-9
    trunc = 5.0 * voxel
    return (-(f - 0.35) / gn).clamp(-trunc, trunc).float().reshape(-1)


def _views(case, seed):
    """Depth views (float64 [h, w], as integrated) of the ellipsoid scene from
    a camera that circles it by a few degrees, with their poses."""
    seq = _sequence("ellipsoids", 256, seed)
    rng = np.random.default_rng(100 + seed)
    rays = synth.pixel_rays()
    centre = np.array([0.0, 0.0, 0.81])
    out = []
    for k in range(case["views"]):
        R = synth.rot(rng.normal(size=3), rng.uniform(0.02, 0.25)) if k else np.eye(3)
        t = centre - R @ centre
        shapes = [synth.Ellipsoid(R.T @ (s.centre - t), s.axes, R.T @ s.R) for s in seq.shapes(0)]
        d = synth.to_frame(synth.render(shapes, rays), seq.sigma, seed, k)
        pose = np.eye(4)
        pose[:3, :3], pose[:3, 3] = R, t
        if case["u16"]:
            d = np.rint(d.astype(np.float64) * 1000.0).astype(np.uint16)
        out.append((d, pose))
    return out


class _DeviceArray:
    """A device array of a grid as torch sees it; a tensor made from it keeps
    the grid alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": typestr,
                                         "version": 3}


def _planes(grid):
    p, w = grid.device_ptrs()
    return (torch.as_tensor(_DeviceArray(grid, p, grid.shape, "<f4"), device=DEV),
            torch.as_tensor(_DeviceArray(grid, w, grid.shape, "<i4"), device=DEV))


def _grid(dims, voxel, origin, P, phi=None, w=None):
    g = capi.Grid(dims, voxel, origin, P.unknown_clip, P)
    if phi is not None:
        if w is None:
            w = (phi <= P.max_surface).to(torch.int32)
        capi.check(capi.load().kf_grid_upload(g.h, phi.data_ptr(), w.data_ptr(), None))
        torch.cuda.synchronize()
    return g


def _read_psi(field, out):
    capi.check(capi.load().kf_field_download(field.h, out.data_ptr(), None))
    return out


def _batch_sizes(case):
    rng = np.random.default_rng(case["problems"])
    return [int(n) for n in rng.integers(case["lo"], case["hi"] + 1, case["problems"])]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        live, can, lw, cw, P, voxel, origin = _scene_sdfs(case, seed)
        dims = _dims(case)
        exact = case["solver"] == "exact"
        return {"case": case, "params": P, "live": _grid(dims, voxel, origin, P, live, lw),
                "can": _grid(dims, voxel, origin, P, can, cw),
                "psi": capi.Field(dims, capi.KF_F64 if exact else capi.KF_F32),
                "out": torch.zeros(dims[::-1] + (3,), device=DEV,
                                   dtype=torch.float64 if exact else torch.float32)}
    if kind == "batch":
        rng, sizes = np.random.default_rng(1000 + seed), _batch_sizes(case)
        problems = []
        out = torch.zeros((sum(n ** 3 for n in sizes), 3), device=DEV)
        for n in sizes:
            can, live, voxel = _shape_sdfs(n, rng)
            P = _params(voxel)
            dims = (n, n, n)
            problems.append((_grid(dims, voxel, (0, 0, 0), P, live), _grid(dims, voxel, (0, 0, 0), P, can),
                             capi.Field(dims), P))
        return {"case": case, "problems": problems, "out": out, "parts": out.split([n ** 3 for n in sizes]),
                "batch": capi.Batch(problems, case["iterations"])}
    if kind == "integrate":
        voxel, origin = _placement(case)
        P = _params(voxel)
        views = [(torch.from_numpy(d.view(np.int16) if case["u16"] else d).to(DEV), pose)
                 for d, pose in _views(case, seed)]
        return {"case": case, "params": P, "views": views, "grid": _grid(_dims(case), voxel, origin, P)}
    if kind == "mesh":
        live, _, lw, _, P, voxel, origin = _scene_sdfs(case, seed)
        dims = _dims(case)
        psi = _solved_psi(case, seed, live, P)
        field = capi.Field(dims)
        capi.check(capi.load().kf_field_upload(field.h, psi.data_ptr(), None))
        torch.cuda.synchronize()
        cap = max(dims) ** 2
        return {"case": case, "params": P, "live": _grid(dims, voxel, origin, P, live, lw), "psi": field,
                "dst": _grid(dims, voxel, origin, P), "cap": cap,
                "verts": torch.zeros((cap, 9), device=DEV),
                "ntri": torch.zeros((1,), dtype=torch.int64, device=DEV)}
    if kind == "energy":
        dims = _dims(case)
        live, can, psi, active, P, voxel = _energy_inputs(case, seed)
        field = capi.Field(dims)
        capi.check(capi.load().kf_field_upload(field.h, psi.data_ptr(), None))
        torch.cuda.synchronize()
        return {"case": case, "params": P, "live": _grid(dims, voxel, (0, 0, 0), P, live),
                "can": _grid(dims, voxel, (0, 0, 0), P, can), "psi": field, "active": active,
                "grad": torch.zeros(dims[::-1] + (3,), dtype=torch.float64, device=DEV)}
    seq = _sequence(case["scene"], case["n"], seed)
    g = seq.grid
    n = max(g.dims)
    frames = [torch.from_numpy(seq.frame(f)).to(DEV) for f in range(case["frames"] + 1)]
    pipe = pipeline.FramePipeline(g.dims, g.voxel, g.origin, _params(g.voxel), case["iterations"],
                                  solver=case["solver"], mesh_capacity=n * n)
    for slot in pipe.meshes:
        for m in slot:
            m.zero_()
    return {"case": case, "pipe": pipe, "frames": frames}


def _solved_psi(case, seed, live, P):
    """psi as a solve leaves it: smooth, up to 1.5 voxels, zero off the band
    (float32 [nz, ny, nx, 3])."""
    dims = _dims(case)
    psi = _smooth_psi(dims, np.random.default_rng(200 + seed), 1.5)
    band = (live <= P.max_surface - P.epsilon) & (live >= -P.unknown_clip)
    return (psi * band.view(dims[::-1] + (1,))).float()


def _energy_inputs(case, seed):
    dims = _dims(case)
    voxel = 0.004
    rng = np.random.default_rng(300 + seed)
    live, can = _blobs(dims, rng, voxel), _blobs(dims, rng, voxel)
    psi = _smooth_psi(dims, rng, 2.0).float()
    P = _params(voxel).with_(gamma_k=0.1)
    active = (live.abs() < P.unknown_clip).to(torch.uint8)
    return live, can, psi, active, P, voxel


def run(s):
    case = s["case"]
    kind = case["kind"]
    L = capi.load()
    if kind == "solve":
        s["psi"].zero()
        st = capi.psi_solve(s["live"], s["can"], s["psi"], s["params"], case["iterations"], case["solver"])
        return [_read_psi(s["psi"], s["out"]), st["iterations_run"], st["active_first"], st["active_last"],
                st["max_delta_last"], st["energy_last"]]
    if kind == "batch":
        for _, _, psi, _ in s["problems"]:
            psi.zero()
        st = s["batch"].run()
        for p, part in zip(s["problems"], s["parts"]):
            _read_psi(p[2], part)
        return [s["out"], np.array([t["active_last"] for t in st]), np.array([t["energy_last"] for t in st])]
    if kind == "integrate":
        g = s["grid"]
        for k, (d, pose) in enumerate(s["views"]):
            if k == 0:
                g.compute_sdf(s["params"], d, pose, u16_scale=0.001 if case["u16"] else None)
            elif case["u16"]:
                g.integrate_u16(d, 0.001, pose)
            else:
                g.integrate(d, pose)
        return list(_planes(g))
    if kind == "mesh":
        P, dst = s["params"], s["dst"]
        dst.reset(P)
        capi.fuse_warped(dst, s["live"], s["psi"], P)
        capi.check(L.kf_marching_cubes_async(dst.h, C.byref(P.c()), s["verts"].data_ptr(), s["cap"],
                                             s["ntri"].data_ptr(), None))
        return list(_planes(dst)) + [s["ntri"], s["verts"]]
    if kind == "energy":
        P, a = s["params"], s["active"].data_ptr()
        terms = np.zeros(3)
        args = (s["live"].h, s["can"].h, s["psi"].h, C.byref(P.c()), a)
        capi.check(L.kf_energy(*args, None, capi.KF_F64, terms.ctypes.data_as(C.POINTER(C.c_double)), None))
        capi.check(L.kf_energy_adjoint(*args, s["grad"].data_ptr(), None))
        return [terms, s["grad"]]
    pipe, frames = s["pipe"], s["frames"]
    pipe.start(frames[0])
    _, tris, _ = pipe.run([(f, frames[f]) for f in range(1, len(frames))], copy=True)
    # every frame's triangle counts, the meshes of the two frames in flight
    # last and the canonical SDF
    return [np.array(tris), pipe.meshes] + list(_planes(pipe.can))


# About how many voxels of an n-voxel-wide depth view's band a solve moves
# (measured: 14 k at 256^3, 0.21 n^2) and float operations of one voxel's
# step (20 neighbours of 3 components, 26 trilinear samples, the terms).
_BAND, _STEP = 0.21, 1500


def work(case):
    kind = case["kind"]
    if kind == "sequence":
        n, its = case["n"], case["iterations"] * case["frames"]
        # per frame: the depth, the live SDF written, the canonical one read
        # and written; the first frame's SDF written
        return {"bytes": (case["frames"] * (8 + 16) + 8) * n ** 3 + (case["frames"] + 1) * 4 * 640 * 480,
                "flops": _BAND * n * n * its * _STEP}
    if kind == "batch":
        sizes = _batch_sizes(case)
        # closed surfaces: a band of about 2.5 n^2 voxels
        return {"bytes": 20 * sum(n ** 3 for n in sizes),
                "flops": sum(2.5 * n * n for n in sizes) * case["iterations"] * _STEP}
    nx, ny, nz = _dims(case)
    N = nx * ny * nz
    if kind == "solve":
        # both SDFs read, psi written once
        size = 8 if case["solver"] == "exact" else 4
        return {"bytes": (8 + 3 * size) * N, "flops": _BAND * max(nx, ny, nz) ** 2 * case["iterations"] * _STEP}
    if kind == "integrate":
        return {"bytes": 8 * N + case["views"] * 640 * 480 * (2 if case["u16"] else 4), "flops": 30 * N}
    if kind == "mesh":
        # psi, the SDF and its weights read; the new SDF and weights written
        return {"bytes": (12 + 8 + 8) * N, "flops": 60 * N}
    # both SDFs, psi and the mask read, the float64 gradient written
    return {"bytes": (8 + 12 + 1 + 24) * N, "flops": 600 * N}


# ---------------------------------------------------------------------------
# the results in 64 bits
# ---------------------------------------------------------------------------

def _lerp(a, b, t):
    return a * (1.0 - t) + b * t


def _trilinear(corner, t):
    """corner(c) -> values at cell corner c = (dx, dy, dz); t: fractions."""
    e = [[_lerp(corner(0, y, z), corner(1, y, z), t[0]) for y in (0, 1)] for z in (0, 1)]
    return _lerp(_lerp(e[0][0], e[0][1], t[1]), _lerp(e[1][0], e[1][1], t[1]), t[2])


def _phi_sample(phi, dims, oob, t):
    """phi (flat) at t = three coordinate tensors, half a voxel already off."""
    nx, ny, nz = dims
    b = [q.trunc() for q in t]
    i = [q.to(torch.int64) for q in b]

    def corner(dx, dy, dz):
        x, y, z = i[0] + dx, i[1] + dy, i[2] + dz
        ok = (x >= 0) & (x < nx) & (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
        return torch.where(ok, phi[torch.where(ok, (z * ny + y) * nx + x, 0)], oob)

    return _trilinear(corner, [t[k] - b[k] for k in range(3)])


def _psi_sample(psi, dims, t):
    """psi ([N, 3]) at t; a linear index off the grid reads 0.  [..., 3]."""
    nx, ny, nz = dims
    N = nx * ny * nz
    b = [q.trunc() for q in t]
    i = [q.to(torch.int64) for q in b]

    def corner(dx, dy, dz):
        k = ((i[2] + dz) * ny + i[1] + dy) * nx + i[0] + dx
        ok = (k >= 0) & (k < N)
        return torch.where(ok[..., None], psi[torch.where(ok, k, 0)], 0.0)

    return _trilinear(corner, [(t[k] - b[k])[..., None] for k in range(3)])


# gradient offsets, then the 19 of the second differences
_OFF = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
        (0, 0, 0), (2, 0, 0), (-2, 0, 0), (0, 2, 0), (0, -2, 0), (0, 0, 2), (0, 0, -2),
        (1, 0, 1), (-1, 0, 1), (0, 1, 1), (0, -1, 1), (1, 1, 0), (-1, 1, 0),
        (-1, 0, -1), (1, 0, -1), (0, -1, -1), (0, 1, -1), (-1, -1, 0), (1, -1, 0)]


def _second(f):
    """xx, yy, zz, xz, yz, xy of the 19 samples f[0..18]."""
    return (f[1] - 2 * f[0] + f[2], f[3] - 2 * f[0] + f[4], f[5] - 2 * f[0] + f[6],
            f[7] + f[13] - f[14] - f[8], f[9] + f[15] - f[16] - f[10], f[11] + f[17] - f[18] - f[12])


def _norm(v):
    return torch.sqrt((v * v).sum(-1))


def _gradient64(live, can, psi, dims, P, idx):
    """KillingFusion::computeEnergyGradient at the voxels idx, the warped
    value s and the monitored energy, float64."""
    nx, ny, _ = dims
    oob, h = P.max_surface + P.epsilon, P.delta_size
    ijk = [idx % nx, (idx // nx) % ny, idx // (nx * ny)]
    x = [q.double() for q in ijk]
    own = psi[idx]
    s = _phi_sample(live, dims, oob, [x[k] + own[:, k] for k in range(3)])
    o = torch.tensor(_OFF, dtype=torch.float64, device=DEV) * h
    at = [x[k][None] + 0.5 + o[:, k, None] for k in range(3)]
    d = _psi_sample(psi, dims, at)
    f = _phi_sample(live, dims, oob, [at[k] + d[..., k] for k in range(3)])
    g = torch.stack([(f[2 * k] - f[2 * k + 1]) / (2 * h) for k in range(3)], -1)
    xx, yy, zz, xz, yz, xy = (q / (4 * h * h) for q in _second(f[6:]))
    gn = _norm(g)
    hg = torch.stack([xx * g[:, 0] + xy * g[:, 1] + xz * g[:, 2], xy * g[:, 0] + yy * g[:, 1] + yz * g[:, 2],
                      xz * g[:, 0] + yz * g[:, 1] + zz * g[:, 2]], -1)
    r = (s - can[idx]) / P.voxel_size
    out = r[:, None] * g + hg * ((gn - 1) / (gn + P.epsilon) * P.omega_s)[:, None]
    kd = _psi_sample(psi, dims, [x[k][None] + o[6:, k, None] for k in range(3)])
    kx, ky, kz, kxz, kyz, kxy = _second(kd)
    div = torch.stack([kx[:, 0] + kxy[:, 1] + kxz[:, 2], kxy[:, 0] + ky[:, 1] + kyz[:, 2],
                       kxz[:, 0] + kyz[:, 1] + kz[:, 2]], -1)
    kg = -2 * (kx + ky + kz) - 2 * P.gamma_k * div
    kn = _norm(kg)[:, None]
    kg = torch.where(kn > P.killing_clamp, kg / kn * P.killing_clamp, kg) / (4 * h * h)
    out = out + kg * P.omega_k
    J = []
    for k in range(3):
        p, m = list(ijk), list(ijk)
        p[k], m[k] = (ijk[k] + 1).clamp(max=dims[k] - 1), (ijk[k] - 1).clamp(min=0)
        lin = lambda q: (q[2] * ny + q[1]) * nx + q[0]  # noqa: E731
        J.append(0.5 * (psi[lin(p)] - psi[lin(m)]))
    J = torch.stack(J, -1)
    e = 0.5 * r * r + P.omega_s * 0.5 * (gn / P.voxel_size - 1) ** 2 + P.omega_k * (
        (J * J).sum((1, 2)) + P.gamma_k * (J * J.transpose(1, 2)).sum((1, 2)))
    return out, s, e


def _chunks(idx, size=1 << 17):
    return idx.split(size) if idx.numel() else []


def _jacobi64(live, can, dims, P, iterations):
    """psi and the last iteration's statistics of the Jacobi schedule.  A
    voxel outside the band keeps psi, so the band only shrinks."""
    live, can = live.double(), can.double()
    N = live.numel()
    psi = torch.zeros((N, 3), dtype=torch.float64, device=DEV)
    in_band = lambda s: ~((s > P.max_surface - P.epsilon) | (s < -P.unknown_clip))  # noqa: E731
    idx = in_band(live).nonzero().reshape(-1)
    first = idx.numel()
    active, maxd, energy = first, 0.0, 0.0
    for it in range(iterations):
        new, keep, es = [], [], []
        for c in _chunks(idx):
            g, s, e = _gradient64(live, can, psi, dims, P, c)
            on = in_band(s)
            keep.append(c[on])
            new.append(-P.alpha * g[on])
            es.append(e[on])
        if not keep:
            break
        idx, d = torch.cat(keep), torch.cat(new)
        psi[idx] += d
        if it == iterations - 1:
            active, maxd = idx.numel(), float(_norm(d).max()) if idx.numel() else 0.0
            energy = float(torch.cat(es).sum())
    return psi, first, active, maxd, energy


def _pervoxel64(live, can, dims, P, cap):
    """The per-voxel schedule, colour by colour (parity of x, y, z)."""
    live, can = live.double(), can.double()
    nx, ny, _ = dims
    psi = torch.zeros((live.numel(), 3), dtype=torch.float64, device=DEV)
    hi = P.max_surface - P.epsilon
    idx = ((live <= hi) & (live >= -hi)).nonzero().reshape(-1)
    color = (idx % nx & 1) | (idx // nx % ny & 1) << 1 | (idx // (nx * ny) & 1) << 2
    for c in range(8):
        cur = idx[color == c]
        for _ in range(cap):
            if cur.numel() == 0:
                break
            g = torch.cat([_gradient64(live, can, psi, dims, P, q)[0] for q in _chunks(cur)])
            psi[cur] += -P.alpha * g
            cur = cur[(_norm(P.alpha * g) > P.threshold) & (_norm(g) > P.threshold)]
    return psi


def _warped_energy64(live, can, psi, active, dims, P):
    """The three energy terms and their gradient with respect to psi."""
    nx, ny, nz = dims
    live, can = live.double(), can.double()
    psi = psi.double().reshape(nz, ny, nx, 3).clone().requires_grad_(True)
    ax = [torch.arange(n, dtype=torch.float64, device=DEV) for n in dims]
    x = [ax[0].view(1, 1, nx), ax[1].view(1, ny, 1), ax[2].view(nz, 1, 1)]
    pw = _phi_sample(live, dims, P.max_surface + P.epsilon, [x[k] + psi[..., k] for k in range(3)])
    on = active.view(nz, ny, nx).double()

    def half_diff(t, axis):
        n = t.shape[axis]
        i = torch.arange(n, device=DEV)
        return 0.5 * (t.index_select(axis, (i + 1).clamp(max=n - 1)) - t.index_select(axis, (i - 1).clamp(min=0)))

    v = P.voxel_size
    data = (0.5 * ((pw - can.view(nz, ny, nx)) / v) ** 2 * on).sum()
    g2 = sum(half_diff(pw, a) ** 2 for a in (2, 1, 0))
    level = (P.omega_s * 0.5 * (torch.sqrt(g2 + (v * P.epsilon) ** 2) / v - 1) ** 2 * on).sum()
    J = torch.stack([half_diff(psi, a) for a in (2, 1, 0)], -1)
    kill = (P.omega_k * ((J * J).sum((-1, -2)) + P.gamma_k * (J * J.transpose(-1, -2)).sum((-1, -2))) * on).sum()
    (grad,) = torch.autograd.grad(data + level + kill, psi)
    return torch.stack([data, level, kill]).detach().cpu().numpy(), grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        live, can, _, _, P, _, _ = _scene_sdfs(case, seed)
        dims = _dims(case)
        if case["solver"] == "pervoxel":
            psi = _pervoxel64(live, can, dims, P, case["iterations"])
            return [psi.view(dims[::-1] + (3,)), None, None, None, None, None]
        psi, _, _, maxd, energy = _jacobi64(live, can, dims, P, case["iterations"])
        if case["solver"] == "exact":  # its statistics are float sums, psi float64
            return [psi.view(dims[::-1] + (3,)), None, None, None, None, None]
        return [psi.view(dims[::-1] + (3,)), None, None, None, maxd, energy]
    if kind == "batch":
        rng, sizes = np.random.default_rng(1000 + seed), _batch_sizes(case)
        if case["iterations"] * sum(n * n for n in sizes) > 1.5e7:
            return None  # above 20 s
        psis, energies = [], []
        for n in sizes:
            can, live, voxel = _shape_sdfs(n, rng)
            psi, _, _, _, e = _jacobi64(live, can, (n, n, n), _params(voxel), case["iterations"])
            psis.append(psi)
            energies.append(e)
        return [torch.cat(psis), None, np.array(energies)]
    if kind == "integrate":
        voxel, origin = _placement(case)
        P = _params(voxel)
        dims = _dims(case)
        n = dims[0] * dims[1] * dims[2]
        phi = torch.full((n,), P.max_surface + P.epsilon, dtype=torch.float64, device=DEV)
        w = torch.zeros_like(phi)
        for d, pose in _views(case, seed):
            d = torch.from_numpy(d.astype(np.float64)).to(DEV) * (0.001 if case["u16"] else 1.0)
            phi, w = _tsdf(phi, w, d, pose, dims, voxel, origin, P.unknown_clip)
        return [phi.view(dims[::-1]), None]
    if kind == "mesh":
        live, _, lw, _, P, _, _ = _scene_sdfs(case, seed)
        dims = _dims(case)
        nx, ny, nz = dims
        psi = _solved_psi(case, seed, live, P).double()
        i = torch.arange(nx * ny * nz, device=DEV)
        x = [(i % nx).double(), (i // nx % ny).double(), (i // (nx * ny)).double()]
        t = [x[k] + 0.5 + psi.view(-1, 3)[:, k] - 0.5 for k in range(3)]
        w = _phi_sample(lw.double(), dims, 0.0, t)
        phi = _phi_sample(live.double(), dims, P.max_surface + P.epsilon, t)
        phi = torch.where(w.abs() < 1e-5, P.max_surface + P.epsilon, phi)
        # the mesh is a list whose length the cases of each cell decide: no
        # 64-bit value of the same layout
        return [phi.view(dims[::-1]), None, None, None]
    if kind == "energy":
        live, can, psi, active, P, _ = _energy_inputs(case, seed)
        terms, grad = _warped_energy64(live, can, psi, active, _dims(case), P)
        return [terms, grad]
    return None  # a chain of solves, truncated weights and meshes
