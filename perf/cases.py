"""The calls whose speed this repository is judged by: sessions stepped frame by frame (small,
headline and large volumes, both trackers, host and device frames, one at a time and batched),
single stages called on their own, mesh extraction and the prefix sum.

Scenes, trajectories and the depth noise model are the package's synthetic sequences; volume
sizes, storages, iteration counts and quirk sets are those of its workloads and tests.  Frame
cases fuse the first frames of a sequence in prepare() and walk the following ones back and
forth, one frame a pass, so that the volume, the pose and the maps are those of a running
session.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from oglfusionkinectv2_b200 import GFusion, GFusionBatch, GFusionConfig, MCubes, _lib as L, prefix_sum_device, synth

STORAGES = {"f32": L.KF_STORAGE_F32F32, "f16": L.KF_STORAGE_F16U16, "rg16i": L.KF_STORAGE_RG16I}
QUIRKS = {"tracking": L.KF_QUIRKS_TRACKING, "default": L.KF_QUIRKS_DEFAULT, "reference": L.KF_QUIRKS_REFERENCE}
FUSED = 4     # frames a session has seen before the first pass
AHEAD = 8     # frames it then walks back and forth
VIEWS = 3     # views of the integrate cases
IR = (365.1, 364.7, 255.3, 208.9, 0.092, -0.27, 0.094, 0.0012, -0.0006)  # a Kinect v2's IR camera
PIXELS = 512 * 424


def listed() -> list[dict]:
    return [
        # the smallest call: a few thousand counts scanned between two kernels of a host program
        {"name": "scan_4k", "kind": "scan", "n": 4099},
        # compaction offsets of a whole 464^3 volume's voxels, an odd length
        {"name": "scan_100m", "kind": "scan", "n": 100_000_007},
        # the mapping stage alone (poses from elsewhere) at the headline volume
        {"name": "integrate_512", "kind": "integrate", "nx": 512, "ny": 512, "nz": 512, "storage": "f16",
         "quirks": "tracking"},
        # the smallest session: 128^3 float, FP32 sums, where launches and hand-overs count
        {"name": "frame_128", "kind": "frame", "nx": 128, "ny": 128, "nz": 128, "storage": "f32", "split_bf16": False,
         "sdf": False, "quirks": "tracking"},
        # the headline: 512^3 over 3 m, half TSDF + uint16 weight, split-BF16 sums, ICP {10, 5, 4}
        {"name": "frame_512", "kind": "frame", "nx": 512, "ny": 512, "nz": 512, "storage": "f16", "split_bf16": True,
         "sdf": False, "quirks": "tracking"},
        # the largest: 768^3 room walk with direct SDF tracking
        {"name": "frame_768_sdf", "kind": "frame", "nx": 768, "ny": 768, "nz": 768, "storage": "f16",
         "split_bf16": False, "sdf": True, "quirks": "tracking"},
        # a camera loop: frames from host memory, pipelined, the previous frame's pose read each call
        {"name": "stream_256", "kind": "stream", "nx": 256, "ny": 256, "nz": 256, "storage": "f16",
         "split_bf16": True, "quirks": "tracking"},
        # the reference application's own loop: raw float depth through undistortion and filter, every
        # stage called by itself with the reference's behaviour and storage, the model read back for
        # display; a ragged volume
        {"name": "view_ragged", "kind": "view", "nx": 250, "ny": 203, "nz": 187, "storage": "rg16i",
         "quirks": "reference"},
        # a server's step: sessions of mixed sizes advanced together
        {"name": "batch_16", "kind": "batch", "sessions": 16, "largest": 384, "storage": "f16", "split_bf16": True},
        # a mesh for display from the headline volume (the reference's extraction), read back
        {"name": "mc_512", "kind": "soup", "nx": 512, "ny": 512, "nz": 512, "storage": "f16", "scan": False,
         "quirks": "tracking"},
        # the classic extraction with normals from a small ragged float volume
        {"name": "mc_scan_ragged", "kind": "soup", "nx": 205, "ny": 160, "nz": 131, "storage": "f32", "scan": True,
         "quirks": "default"},
        # an indexed mesh for export
        {"name": "mesh_384", "kind": "mesh", "nx": 384, "ny": 384, "nz": 384, "storage": "f16", "quirks": "tracking"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["scan", "integrate", "frame", "stream", "view", "batch", "soup", "mesh"])
    if kind == "scan":
        return {"kind": kind, "n": _log_int(rng, 1, 100_000_007)}
    quirks = rng.choice(["tracking", "default", "reference"])
    if kind == "batch":
        return {"kind": kind, "sessions": rng.randint(2, 16), "largest": rng.choice([128, 192, 256, 384]),
                "storage": rng.choice(["f16", "f32"]), "split_bf16": rng.random() < 0.7}
    most = {"frame": 600, "stream": 512, "view": 384}.get(kind, 512)
    side = _log_int(rng, 64, most)
    case = {"kind": kind}
    for axis in ("nx", "ny", "nz"):  # cubes as often as ragged volumes
        case[axis] = side if rng.random() < 0.7 else rng.randint(max(48, side // 2), side)
    case["storage"] = rng.choice(["f32", "f16", "rg16i"])
    case["quirks"] = quirks
    if kind in ("frame", "stream"):
        case["split_bf16"] = rng.random() < 0.5
        if kind == "frame":
            case["sdf"] = rng.random() < 0.3
    if kind == "soup":
        case["scan"] = rng.random() < 0.5
    return case


# ---- inputs -----------------------------------------------------------------------------------
def _size(case) -> tuple:
    return case["nx"], case["ny"], case["nz"]


def _workload(case, seed: int, frames: int):
    """The synthetic sequence of a case: the room walk for SDF tracking, else spheres and boxes
    on a ground plane seen from an orbit (1.5 m volumes up to 256 voxels, 3 m above)."""
    side = max(_size(case))
    seed = synth.splitmix64(seed * 7919 + 17) & 0xFFFFFFFF
    if case.get("sdf"):
        w = synth.large_c5(frames, seed=seed, size=side)
    elif side <= 256:
        w = synth.session_scene(frames, seed, side)
    else:
        w = synth.precision_c2(frames, seed=seed, size=side)
    c = w.config
    c.volumeSize = _size(case)
    c.storage = STORAGES[case["storage"]]
    c.quirks = QUIRKS[case.get("quirks", "tracking")]
    c.jtj = L.KF_JTJ_SPLIT_BF16 if case.get("split_bf16") else L.KF_JTJ_FP32
    return w


def _walk(n: int, k: int) -> int:
    """k-th index of 0, 1, ..., n-1, n-2, ..., 1, 0, 1, ..."""
    p = 2 * (n - 1)
    k %= p
    return k if k < n else p - k


class _Span:
    """A stretch of a session's device memory as torch sees it; the session lives as long."""

    def __init__(self, owner: GFusion, ptr: int, shape: tuple, kind: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}


def _volume(g: GFusion) -> dict:
    """The session's own value and weight planes, as tensors."""
    v = g.getVolumeView()
    shape = (v.nz, v.ny, v.nx)
    kinds = {L.KF_STORAGE_F32F32: ("<f4", "<f4"), L.KF_STORAGE_F16U16: ("<f2", "<i2"), L.KF_STORAGE_RG16I: ("<i2", "<i2")}
    a, b = kinds[v.storage]
    return {"value": torch.as_tensor(_Span(g, v.device_ptr, shape, a), device="cuda"),
            "weight": torch.as_tensor(_Span(g, v.device_ptr + v.weight_offset_bytes, shape, b), device="cuda")}


def _frames(w, count: int) -> torch.Tensor:
    return w.frames_torch(list(range(count)), "cuda")


def _host(frames: torch.Tensor) -> np.ndarray:
    return frames.cpu().numpy().view(np.uint16)


def _surface_volume(case, seed: int):
    """The TSDF of a whole scene, as a finished scan leaves it: truncated distances with fusion
    noise in the band, zero (nothing observed) deeper than mu inside the objects.  The scene and
    the noise of its surface are the size's own; the seed scales every distance by up to a fifth
    either way, so every seed has its own vertices on the same cubes.  Returns the configuration
    and the stored values, exactly representable in the storage."""
    w = _workload(case, max(_size(case)), 1)
    c = w.config
    nx, ny, nz = c.volumeSize
    d = c.volumeDimensions
    ax = [(torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * (d[k] / n) for k, n in enumerate((nx, ny, nz))]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    f = (w.scene.planes[0][1] - Y).expand(nz, ny, nx).clone()
    for (cx, cy, cz), r in w.scene.spheres:
        f = torch.minimum(f, ((X - cx) ** 2 + (Y - cy) ** 2 + (Z - cz) ** 2).sqrt() - r)
    for lo, hi in w.scene.boxes:
        q = [torch.clamp(torch.maximum(lo[k] - a, a - hi[k]), min=-1.0) for k, a in enumerate((X, Y, Z))]
        f = torch.minimum(f, torch.maximum(torch.maximum(q[0], q[1]), q[2]))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(max(_size(case)))
    f = f / c.mu
    f += 0.05 * torch.randn(f.shape, generator=gen, device="cuda")
    # distances too small for the fixed-point storage's sign are pushed off zero
    f = torch.where(f.abs() < 1e-3, torch.copysign(torch.full_like(f, 1e-3), f), f)
    f = torch.where(f > -1.0, f, torch.zeros_like(f))
    gen.manual_seed(seed)
    f *= 0.8 + 0.4 * torch.rand(f.shape, generator=gen, device="cuda")
    f = f.clamp(-1.0, 1.0)
    if c.storage == L.KF_STORAGE_F16U16:
        f = f.half()
    elif c.storage == L.KF_STORAGE_RG16I:
        f = (f * 32766.0).to(torch.int16)
    return c, w.intrinsics, f


def _with_volume(case, seed: int) -> GFusion:
    c, intr, f = _surface_volume(case, seed)
    g = GFusion(c, intr)
    raw = f.cpu().numpy().reshape(-1).view(np.uint8)
    wt = (np.full(f.numel(), 20, np.float32) if c.storage == L.KF_STORAGE_F32F32 else np.full(f.numel(), 20, np.int16))
    g.setVolumeRaw(np.concatenate([raw, wt.view(np.uint8)]))
    return g


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "scan":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        # triangle counts: mostly zero, at most 5
        x = torch.randint(0, 6, (case["n"],), generator=gen, device="cuda", dtype=torch.int32)
        x *= torch.rand(case["n"], generator=gen, device="cuda") < 0.3
        return {"kind": kind, "in": x, "out": torch.empty_like(x)}
    if kind in ("soup", "mesh"):
        g = _with_volume(case, seed)
        m = MCubes(g)
        m.setIsolevel(0.0)
        return {"kind": kind, "g": g, "mc": m, "method": L.KF_MC_SCAN if case.get("scan") else L.KF_MC_HISTOPYRAMID,
                "normals": bool(case.get("scan"))}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        mix = np.random.default_rng(case["sessions"])  # the sizes are the case's, the scenes the seed's
        sizes = [s for s in synth.C3_SIZES if s <= case["largest"]]
        sessions, frames = [], []
        for k in range(case["sessions"]):
            size = case["largest"] if k == 0 else int(mix.choice(sizes))
            w = synth.session_scene(FUSED + AHEAD, int(rng.integers(1 << 31)), size, float(rng.uniform(0.0, 360.0)),
                                    0.5 if rng.random() < 0.5 else -0.5)
            w.config.storage = STORAGES[case["storage"]]
            w.config.jtj = L.KF_JTJ_SPLIT_BF16 if case["split_bf16"] else L.KF_JTJ_FP32
            g = GFusion(w.config, w.intrinsics)
            g.Reset(w.poses[0])
            sessions.append(g)
            frames.append(_frames(w, FUSED + AHEAD))
        torch.cuda.synchronize()
        b = GFusionBatch(len(sessions))
        for k in range(FUSED):
            b.frameStepDevice(sessions, [f[k].data_ptr() for f in frames])
        return {"kind": kind, "b": b, "g": sessions, "frames": frames, "k": 0}
    if kind == "integrate":
        w = _workload(case, seed, 40)
        views = [k * 39 // (VIEWS - 1) for k in range(VIEWS)]
        frames = _host(w.frames_torch(views, "cuda"))
        g = GFusion(w.config, w.intrinsics)
        g.Reset(w.poses[0])
        for j, k in enumerate(views):
            g.setPose(w.poses[k])
            g.depthToVertex(frames[j])
            if j < VIEWS - 1:
                g.integrate()
        return {"kind": kind, "g": g}
    w = _workload(case, seed, FUSED + AHEAD)
    frames = _frames(w, FUSED + AHEAD)
    torch.cuda.synchronize()
    g = GFusion(w.config, w.intrinsics)
    g.Reset(w.poses[0])
    state = {"kind": kind, "g": g, "k": 0}
    if kind == "frame":
        for k in range(FUSED):
            g.frameStepDevice(frames[k].data_ptr())
        state["frames"] = frames
        return state
    host = torch.empty(frames.shape, dtype=torch.int16, pin_memory=True)
    host.copy_(frames)
    host = host.numpy().view(np.uint16)
    if kind == "stream":
        for k in range(FUSED):
            g.frameStepAsync(host[k])
        g.frameSync()
        state["frames"] = host
        return state
    state["frames"] = [f.astype(np.float32) for f in host]
    g.setDepthUndistortion(IR)
    g.setDepthFilter(True)
    for k in range(FUSED):
        _one_view(g, state["frames"][k], first=(k == 0))
    return state


def _one_view(g: GFusion, depth: np.ndarray, first: bool = False) -> bool:
    g.depthToVertex(depth)
    g.vertexToNormal()
    tracked = g.Track()
    if tracked or first:
        g.integrate()
    g.raycast()
    return tracked


def run(state: dict):
    kind = state["kind"]
    if kind == "scan":
        x = state["in"]
        stream = torch.cuda.current_stream().cuda_stream
        total = prefix_sum_device(x.data_ptr(), state["out"].data_ptr(), x.numel(), stream)
        return {"sums": state["out"], "total": total}
    if kind == "soup":
        m = state["mc"]
        out = {"triangles": m.generateMarchingCubes(state["method"]), "vertices": m.getVertices()}
        if state["normals"]:
            out["normals"] = m.getNormals()
        return out
    if kind == "mesh":
        p, n, i = state["mc"].extractMesh()
        return {"positions": p, "normals": n, "indices": i}
    if kind == "integrate":
        state["g"].integrate()
        return _volume(state["g"])
    k = FUSED + _walk(AHEAD, state["k"])
    state["k"] += 1
    if kind == "batch":
        b, sessions = state["b"], state["g"]
        tracked = b.frameStepDevice(sessions, [f[k].data_ptr() for f in state["frames"]])
        return {"tracked": tracked, "poses": b.poses(len(sessions)), "volumes": [_volume(g) for g in sessions]}
    g = state["g"]
    if kind == "frame":
        tracked = g.frameStepDevice(state["frames"][k].data_ptr())
        return {"tracked": tracked, "pose": g.lastResult()[0], **_volume(g)}
    if kind == "stream":
        g.frameStepAsync(state["frames"][k])
        pose, tracked = g.lastResult()
        return {"tracked": tracked, "pose": pose, **_volume(g)}
    tracked = _one_view(g, state["frames"][k])
    return {"tracked": tracked, "pose": g.getPose(), "verts": g.getVerts(), "norms": g.getNorms(), **_volume(g)}


# ---- what a pass cannot do without --------------------------------------------------------------
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "scan":
        return {"bytes": 8 * case["n"], "flops": case["n"]}
    value = 4 if case["storage"] == "f32" else 2
    if kind == "batch":
        one = {"kind": "frame", "nx": 200, "ny": 200, "nz": 200, "storage": case["storage"], "sdf": False}
        w = work(one)
        return {k: v * case["sessions"] for k, v in w.items()}
    n = case["nx"] * case["ny"] * case["nz"]
    surface = 5.0 * n ** (2.0 / 3.0)  # voxels the surface crosses
    if kind in ("soup", "mesh"):
        # the values once; about a triangle per `surface` voxel: 48 bytes of vertices (as much again
        # of normals with the scan path), or 12 of a welded mesh's indices and its vertices' share
        out = 18.0 if kind == "mesh" else 48.0 * (2 if case["scan"] else 1)
        return {"bytes": value * n + out * surface, "flops": 20.0 * surface}
    # the voxels a view updates (free space before the surface and the band behind it, about 4 % of
    # the volume), value and weight read and written, and the depth frame
    touched = 0.04 * n
    b = 4.0 * value * touched + 4 * PIXELS
    f = 40.0 * touched
    if kind == "integrate":
        return {"bytes": b, "flops": f}
    # the frame in, three levels of maps, the raycast maps out
    b += 2 * PIXELS + 36 * PIXELS * 1.3125 + 32 * PIXELS
    # Gauss-Newton: ten fine, five middle, four coarse iterations of ~100 operations a pixel
    f += 100.0 * PIXELS * (10 + 5 / 4 + 4 / 16)
    if kind == "view":
        b += 2 * PIXELS + 32 * PIXELS
    return {"bytes": b, "flops": f}


# ---- the same outputs in 64 bits, by torch alone -------------------------------------------------
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "scan":
        return None  # whole numbers
    if kind == "mesh":
        return _exact_mesh(case, seed)
    if kind == "integrate" and case["storage"] != "rg16i":
        return {"value": _exact_integrate(case, seed), "weight": None}
    # a tracked frame, a soup in the case tables' order, or fixed-point storage: no such value
    return None


def _exact_integrate(case: dict, seed: int) -> torch.Tensor:
    """integrate.cs in 64 bits: the running average of the VIEWS frames at their true poses."""
    w = _workload(case, seed, 40)
    views = [k * 39 // (VIEWS - 1) for k in range(VIEWS)]
    frames = w.frames_torch(views, "cuda").to(torch.float64)
    c, cam = w.config, w.intrinsics
    nx, ny, nz = c.volumeSize
    vs = [c.volumeDimensions[k] / n for k, n in enumerate((nx, ny, nz))]
    f8 = {"dtype": torch.float64, "device": "cuda"}
    X = ((torch.arange(nx, **f8) + 0.5) * vs[0])[None, None, :]
    Y = ((torch.arange(ny, **f8) + 0.5) * vs[1])[None, :, None]
    narrow = bool(c.quirks & L.KF_Q8_NARROW_BAND)
    out = torch.empty((nz, ny, nx), **f8)
    step = max(1, (1 << 23) // (nx * ny))
    for z0 in range(0, nz, step):
        Z = ((torch.arange(z0, min(nz, z0 + step), **f8) + 0.5) * vs[2])[:, None, None]
        F = torch.zeros((Z.shape[0], ny, nx), **f8)
        W = torch.zeros_like(F)
        for j, k in enumerate(views):
            inv = np.linalg.inv(w.poses[k])
            p = [inv[r, 0] * X + inv[r, 1] * Y + inv[r, 2] * Z + inv[r, 3] for r in range(3)]
            pz = p[2]
            u = cam.fx * p[0] / pz + cam.cx + 0.5
            v = cam.fy * p[1] / pz + cam.cy + 0.5
            ok = (pz >= 1e-4) & (u >= 0) & (u <= cam.width - 1) & (v >= 0) & (v <= cam.height - 1)
            at = (torch.where(ok, v, 0.0).long() * cam.width + torch.where(ok, u, 0.0).long())
            d = frames[j].reshape(-1)[at] * 1e-3
            ok &= d != 0
            eta = (d - pz) * (1 + (p[0] / pz) ** 2 + (p[1] / pz) ** 2).sqrt()
            mean = (W * F + torch.clamp(eta / c.mu, max=1.0)) / (W + 1)
            keep = ok & (eta > -c.mu)
            if narrow:
                keep &= mean < 0.2
                mean = mean.clamp(-0.1, 0.2)
            else:
                mean = mean.clamp(-1.0, 1.0)
            F = torch.where(keep, mean, torch.where(ok, 0.0, F))
            W = torch.where(keep, (W + 1).clamp(max=c.maxWeight), torch.where(ok, 0.0, W))
        out[z0:z0 + F.shape[0]] = F
    return out


def _exact_mesh(case: dict, seed: int) -> dict:
    """The welded mesh's vertices in 64 bits: one per cut voxel edge of a cube with a positive
    corner, in voxel order then axis; the unit gradient interpolated along the edge."""
    c, _, f = _surface_volume(case, seed)
    f = f.to(torch.float64)
    nz, ny, nx = f.shape
    first_seven = bool(c.quirks & L.KF_Q13_MC_FIRST_SEVEN)
    # cubes in the classic corner order; corner 7 is (0, 1, 1) in (x, y, z)
    pos = torch.zeros((nz - 1, ny - 1, nx - 1), dtype=torch.bool, device=f.device)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                if not (first_seven and (dx, dy, dz) == (0, 1, 1)):
                    pos |= f[dz:nz - 1 + dz, dy:ny - 1 + dy, dx:nx - 1 + dx] > 0
    neg = f < 0
    used = torch.zeros((nz, ny, nx, 3), dtype=torch.bool, device=f.device)
    for axis in range(3):
        d = 2 - axis  # tensor dimension of the axis
        n = f.shape[d]
        cut = neg.narrow(d, 0, n - 1) != neg.narrow(d, 1, n - 1)
        # an edge belongs to the four cubes around it
        near = torch.zeros_like(cut)
        others = [k for k in range(3) if k != d]
        for s0 in (0, 1):
            for s1 in (0, 1):
                t = near.narrow(others[0], s0, f.shape[others[0]] - 1).narrow(others[1], s1, f.shape[others[1]] - 1)
                t |= pos
        used[..., axis].narrow(d, 0, n - 1).copy_(cut & near)
    at = used.nonzero()
    z, y, x, axis = at.unbind(1)
    size = torch.tensor([nx, ny, nz], device=f.device)
    dim = torch.tensor(c.volumeDimensions, dtype=torch.float64, device=f.device)
    p0 = torch.stack([x, y, z], 1)
    p1 = p0 + torch.nn.functional.one_hot(axis, 3)

    def value(p):
        p = torch.minimum(torch.clamp(p, min=0), size - 1)
        return f[p[:, 2], p[:, 1], p[:, 0]]

    def gradient(p):
        e = torch.eye(3, dtype=torch.int64, device=f.device)
        return torch.stack([(value(p + e[k]) - value(p - e[k])) * (0.5 * size[k] / dim[k]) for k in range(3)], 1)

    f0, f1 = value(p0), value(p1)
    t = ((0.0 - f0) / (f1 - f0))[:, None]
    pts = (p0 + t * (p1 - p0) + 0.5) * dim / size
    g0, g1 = gradient(p0), gradient(p1)
    g = g0 + t * (g1 - g0)
    ln = g.norm(dim=1, keepdim=True)
    nrm = torch.where(ln > 0, g / ln, torch.zeros_like(g))
    return {"positions": pts, "normals": nrm, "indices": None}
