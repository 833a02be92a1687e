"""The work that users of this framework have it do, as cases to be measured.

A case is one call pattern of the public Python API over one size:

live      one depth frame integrated into a volume as it arrives (TSDFVolume.integrate, the reference's per-frame loop)
sequence  a recording integrated in passes of 16 frames (reset, integrate_sequence)
scan      a long recording of one volume through the batched launches (reset, BatchIntegrator.integrate)
scenes    several volumes of different sizes through the same batched launches
mesh      the triangle soup of an integrated volume (extract_mesh_device)
indexed   its mesh with shared vertices and normals (extract_mesh_indexed)
diff      a training step of the differentiable integrate: forward, loss against a model volume, adjoint
cloud     depth and colour frames back-projected into a point cloud, which is then transformed
project   a point cloud projected to a camera's depth and colour images

Scenes are the repository's synthetic ones: a plane and spheres seen from a helix around them, or from poses jittered
about the first camera ("frontal", the reference example's set-up); depth in millimetres (uint16) or metres (float32)
with noise and dropped pixels.  Everything random comes from the seed, but for the volumes that are meshed: they hold
one recording, whose observed distances the seed scales voxel by voxel, so that the triangles stay as many.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cu-reconstruction_gb300"))

from cuphoto import (PointCloud, TSDFVolume, TSDFVolumeConfig, extract_mesh_device,  # noqa: E402
                     extract_mesh_indexed)
from cuphoto import diff as gdiff  # noqa: E402
from cuphoto import synthetic as S  # noqa: E402
from cuphoto.batch import BatchIntegrator  # noqa: E402

CAMERAS = {"qvga": S.Camera.half(), "vga": S.Camera(), "hd": S.Camera.hd()}
DEV = "cuda"


def _case(name, kind, nx=0, ny=0, nz=0, frames=1, camera="vga", depth="u16", mode="compat", arith="reference",
          path="frontal", scenes=1, dtype="f32", colour=True):
    c = dict(kind=kind, frames=frames, camera=camera, depth=depth, path=path)
    if kind in ("cloud", "project"):
        c["colour"] = colour
    elif kind == "diff":
        c.update(nx=nx, ny=ny, nz=nz, dtype=dtype)
        del c["depth"]
    elif kind == "scenes":
        c.update(nx=nx, ny=ny, nz=nz, scenes=scenes, mode=mode, arith=arith)
    else:
        c.update(nx=nx, ny=ny, nz=nz, mode=mode, arith=arith)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a preview volume fed by a small camera: the smallest call, all latency
        _case("live_64", "live", 64, 64, 64, camera="qvga"),
        # the default configuration's grid, frame by frame, depth in metres as the reference passes it
        _case("live_256", "live", 256, 256, 256, depth="f32"),
        # a room at 5 mm, frame by frame, in the corrected mode
        _case("live_512_fixed", "live", 512, 512, 512, mode="fixed", path="helix"),
        # a short recording with odd extents (rows that no vector load fits), correctly rounded arithmetic
        _case("sequence_250", "sequence", 250, 187, 253, frames=32, depth="f32", arith="ieee"),
        # the headline workload: 300 frames into 512^3
        _case("scan_512", "scan", 512, 512, 512, frames=300, path="helix"),
        # a set of objects scanned together, grids of many sizes, corrected mode
        _case("scenes_8", "scenes", 256, 256, 256, frames=60, camera="qvga", mode="fixed", path="helix", scenes=8),
        # the mesh of a large volume
        _case("mesh_512", "mesh", 512, 512, 512, frames=24, mode="fixed", path="helix"),
        # the mesh that is written to a file: shared vertices and normals
        _case("indexed_384", "indexed", 384, 384, 384, frames=24, mode="fixed", path="helix"),
        # a pose-refinement step over the differentiable configuration (128^3, 16 frames 320x240)
        _case("diff_128", "diff", 128, 128, 128, frames=16, camera="qvga", path="helix"),
        # a gradient check in double, more frames than one chunk, odd extents
        _case("diff_45_f64", "diff", 45, 41, 52, frames=11, camera="qvga", path="helix", dtype="f64"),
        # a coloured cloud of eight frames, moved to another coordinate system
        _case("cloud_8", "cloud", frames=8, path="helix"),
        # the cloud of a recording seen from a new viewpoint
        _case("project_30", "project", frames=30, path="helix"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, lo, hi):
    """Three extents of a grid around one size; two thirds of the grids have rows of whole 16-byte vectors."""
    n = _logint(rng, lo, hi)
    e = [max(2, min(hi, int(n * rng.uniform(0.75, 1.25)))) for _ in range(3)]
    if rng.random() < 0.67:
        e[0] = max(4, e[0] // 4 * 4)
    return e


def draw(rng):
    kind = rng.choice(["live", "live", "sequence", "scan", "scenes", "mesh", "indexed", "diff", "cloud", "project"])
    camera = rng.choice(["qvga", "vga", "vga", "hd"])
    path = rng.choice(["helix", "frontal"])
    depth = rng.choice(["u16", "f32"])
    mode, arith = rng.choice([("compat", "reference"), ("compat", "reference"), ("compat", "ieee"), ("fixed", "ieee")])
    if kind == "live":
        return _case("", kind, *_extents(rng, 32, 512), camera=camera, depth=depth, mode=mode, arith=arith, path=path)
    if kind == "sequence":
        return _case("", kind, *_extents(rng, 48, 384), frames=_logint(rng, 8, 64), camera=camera, depth=depth,
                     mode=mode, arith=arith, path=path)
    if kind == "scan":
        return _case("", kind, *_extents(rng, 96, 448), frames=_logint(rng, 40, 200), depth=depth, mode=mode,
                     arith=arith, path=path, camera=rng.choice(["qvga", "vga"]))
    if kind == "scenes":
        return _case("", kind, *_extents(rng, 64, 256), frames=_logint(rng, 10, 60), camera="qvga", depth=depth,
                     mode=mode, arith=arith, path=path, scenes=rng.randint(2, 10))
    if kind in ("mesh", "indexed"):
        if kind == "indexed":
            mode, arith = "fixed", "ieee"
        if mode == "compat":   # whose mesh comes from the grid's first layers: only the frontal set-up has a surface there
            path = "frontal"
        return _case("", kind, *_extents(rng, 40, 512 if kind == "mesh" else 400), frames=_logint(rng, 4, 32),
                     camera="vga", depth=depth, mode=mode, arith=arith, path=path)
    if kind == "diff":
        if rng.random() < 0.25:
            return _case("", kind, *_extents(rng, 20, 64), frames=_logint(rng, 2, 24), camera="qvga", path=path,
                         dtype="f64")
        return _case("", kind, *_extents(rng, 32, 192), frames=_logint(rng, 2, 32),
                     camera=rng.choice(["qvga", "vga"]), path=path)
    return _case("", kind, frames=_logint(rng, 1, 30), camera=camera, depth=depth, path=path,
                 colour=rng.random() < 0.6)


# ---------------------------------------------------------------------------
# Inputs.

def _poses(case, seed, n):
    return S.frontal_poses(n, seed=seed) if case["path"] == "frontal" else S.helix_poses(n, seed=seed)


def _grid(case, extents=None):
    nx, ny, nz = extents or (case["nx"], case["ny"], case["nz"])
    if case["path"] == "frontal":
        return S.frontal_grid(nx, ny, nz)
    return dict(voxel_grid_size=(nx, ny, nz), physical_size=(2.56,) * 3, global_offset=(-1.28,) * 3)


def _frames(case, seed, n):
    """(n, H, W) depth frames (int16 holding uint16 bits, or float32 metres) and their poses."""
    scene = S.make_frontal_scene(seed) if case["path"] == "frontal" else S.make_scene(seed)
    poses = _poses(case, seed, n)
    raw = S.render_sequence_torch(scene, poses, CAMERAS[case["camera"]], seed=seed)
    if case.get("depth", "f32") == "f32":
        raw = (raw.to(torch.int32) & 0xFFFF).float() * np.float32(0.001)
    return raw, poses


def _volume(case, extents=None):
    cam = CAMERAS[case["camera"]]
    return TSDFVolume(TSDFVolumeConfig(**_grid(case, extents), focal_x=cam.fx, focal_y=cam.fy, cx=cam.cx, cy=cam.cy,
                                       camera_width=cam.width, camera_height=cam.height, mode=case["mode"],
                                       arith=case["arith"]))


def _scene_extents(case, k):
    """Scene k's grid: the largest for k = 0, the others from a quarter of it upwards, rows of whole vectors."""
    rng = np.random.default_rng(77 + k)
    f = 1.0 if k == 0 else rng.uniform(0.25, 1.0)
    e = [max(8, int(case[a] * f * rng.uniform(0.8, 1.0))) for a in ("nx", "ny", "nz")]
    e[0] = max(8, e[0] // 4 * 4)
    return e


def _scene_frames(case, k):
    return case["frames"] if k == 0 else max(2, int(case["frames"] * np.random.default_rng(99 + k).uniform(0.2, 1.0)))


def _sdf(case, seed, dtype):
    """Analytic truncated distances of the scene at the voxel centres (z, y, x) and the truncation (4 voxels)."""
    scene = S.make_frontal_scene(seed) if case["path"] == "frontal" else S.make_scene(seed)
    g = _grid(case)
    vs = [np.float32(p) / np.float32(n) for p, n in zip(g["physical_size"], g["voxel_grid_size"])]
    trunc = float(np.float32(4 * max(vs)))
    x, y, z = [(torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * float(v) + o
               for n, v, o in zip(g["voxel_grid_size"], vs, g["global_offset"])]
    d = (scene.plane_up * (y - scene.plane_y))[None, :, None].expand(len(z), len(y), len(x))
    for c, r in zip(scene.centres, scene.radii):
        q = (x - c[0])[None, None, :] ** 2 + (y - c[1])[None, :, None] ** 2 + (z - c[2])[:, None, None] ** 2
        d = torch.minimum(d, q.sqrt() - r)
    return d.clamp(-trunc, trunc).to(dtype), trunc


def _diff_inputs(case, seed):
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    cam = CAMERAS[case["camera"]]
    depth, poses = _frames(case, seed, case["frames"])
    R = np.stack([S.matrix_from_quat(p[:4]) for p in poses])
    t = np.stack([p[4:] for p in poses])
    R, t = S.jitter_poses(R, t, range(len(poses)), 0.5, 0.003, seed)   # poses that are still to be refined
    model, trunc = _sdf(case, seed, dtype)
    g = _grid(case)
    vs = tuple(float(np.float32(p) / np.float32(n)) for p, n in zip(g["physical_size"], g["voxel_grid_size"]))
    cfg = gdiff.DiffConfig(g["voxel_grid_size"], vs, g["global_offset"], cam.fx, cam.fy, cam.cx, cam.cy, trunc,
                           max_weight=128.0, max_depth=8.0, min_z=0.05)
    shape = (case["nz"], case["ny"], case["nx"])
    return dict(depth=depth.to(dtype), R=torch.tensor(R, dtype=dtype, device=DEV),
                t=torch.tensor(t, dtype=dtype, device=DEV), D0=torch.full(shape, trunc, dtype=dtype, device=DEV),
                W0=torch.zeros(shape, dtype=dtype, device=DEV), model=model,
                mask=(model.abs() < 0.999 * trunc).to(dtype), cfg=cfg)


def _colours(frames, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    return torch.randint(0, 256, tuple(frames.shape) + (3,), generator=gen, device=DEV, dtype=torch.uint8)


def _camera_matrix(camera, column_major):
    """cudaPointCloud reads its matrix column-major when back-projecting and row-major when projecting."""
    c = CAMERAS[camera]
    m = [c.fx, 0.0, c.cx, 0.0, c.fy, c.cy, 0.0, 0.0, 1.0]
    return [m[0], m[3], m[6], m[1], m[4], m[7], m[2], m[5], m[8]] if column_major else m


def _inverse(pose):
    R = S.matrix_from_quat(np.asarray(pose[:4], np.float64))
    return S.pose7(R.T, -R.T @ np.asarray(pose[4:], np.float64))


def prepare(case, seed):
    seed = int(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "live":
        depths, poses = _frames(case, seed, 8)
        vol = _volume(case)
        cam = CAMERAS[case["camera"]]
        s.update(vol=vol, depths=list(depths), poses=list(poses), k=0,
                 colour=torch.zeros((cam.height, cam.width, 3), dtype=torch.uint8, device=DEV),
                 out=[vol.voxel_distances_data(), vol.voxel_weights_data()])
    elif kind in ("sequence", "scan"):
        depths, poses = _frames(case, seed, case["frames"])
        vol = _volume(case)
        s.update(vol=vol, depths=depths, poses=list(poses), out=[vol.voxel_distances_data(), vol.voxel_weights_data()])
        if kind == "scan":
            s["batch"] = BatchIntegrator(1, case["frames"])
    elif kind == "scenes":
        n = case["scenes"]
        vols = [_volume(case, _scene_extents(case, k)) for k in range(n)]
        fr = [_frames(case, seed * 16 + k, _scene_frames(case, k)) for k in range(n)]
        s.update(vols=vols, depths=[f[0] for f in fr], poses=[f[1] for f in fr],
                 out=[x for v in vols for x in (v.voxel_distances_data(), v.voxel_weights_data())],
                 batch=BatchIntegrator(n, sum(len(f[1]) for f in fr)))
    elif kind in ("mesh", "indexed"):
        depths, poses = _frames(case, 3, case["frames"])
        vol = _volume(case)
        vol.integrate_sequence(depths, list(poses))
        D, W = vol.voxel_distances_data(), vol.voxel_weights_data()
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        D.mul_(torch.where(W > 0, 0.9 + 0.2 * torch.rand(D.shape, generator=gen, device=DEV), torch.ones_like(D)))
        s["vol"] = vol
    elif kind == "diff":
        s.update(_diff_inputs(case, seed))
        for k in ("depth", "R", "t"):
            s[k].requires_grad_(True)
    elif kind in ("cloud", "project"):
        depths, poses = _frames(case, seed, case["frames"])
        colours = _colours(depths, seed) if case["colour"] else None
        H, W = depths.shape[1:]
        pc = PointCloud.create(_camera_matrix(case["camera"], True), len(depths) * H * W)
        s.update(pc=pc, depths=list(depths), colours=list(colours) if case["colour"] else [None] * len(depths),
                 poses=[_inverse(p) for p in poses], world=S.pose7(*S.look_at((0.4, 0.3, -2.0))))
        if kind == "project":
            for f in range(len(depths)):
                pc.extract_points(s["depths"][f], s["colours"][f], s["poses"][f], f)
            pc.camera_matrix = _camera_matrix(case["camera"], False)
            del s["depths"], s["colours"]
            s["view"] = _poses(case, seed + 1, 3)[1]
            s["image"] = torch.empty((H, W), dtype=torch.float32, device=DEV)
            s["colour"] = torch.empty((H, W, 3), dtype=torch.uint8, device=DEV) if case["colour"] else None
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s["kind"]
    if kind == "live":
        k = s["k"]
        s["k"] = (k + 1) % len(s["depths"])
        s["vol"].integrate(s["colour"], s["depths"][k], s["poses"][k])
        return s["out"]
    if kind == "sequence":
        s["vol"].reset()
        s["vol"].integrate_sequence(s["depths"], s["poses"])
        return s["out"]
    if kind == "scan":
        s["vol"].reset()
        s["batch"].integrate([s["vol"]], [s["depths"]], [s["poses"]])
        return s["out"]
    if kind == "scenes":
        for v in s["vols"]:
            v.reset()
        s["batch"].integrate(s["vols"], s["depths"], s["poses"])
        return s["out"]
    if kind == "mesh":
        return list(extract_mesh_device(s["vol"]))
    if kind == "indexed":
        return list(extract_mesh_indexed(s["vol"]))
    if kind == "diff":
        D, W = gdiff.integrate(s["depth"], s["R"], s["t"], s["D0"], s["W0"], s["cfg"])
        cw = s["mask"] * W
        loss = (cw * (D - s["model"]) ** 2).sum() / cw.sum()
        g = torch.autograd.grad(loss, (s["depth"], s["R"], s["t"]))
        return [D.detach(), W.detach(), loss.detach()] + list(g)
    pc = s["pc"]
    if kind == "cloud":
        pc.clear()
        for f, d in enumerate(s["depths"]):
            pc.extract_points(d, s["colours"][f], s["poses"][f], f)
        pc.transform(s["world"])
        return [pc.get_points()]
    if s["colour"] is None:
        pc.project_to_depth(s["image"], s["view"])
        return [s["image"]]
    pc.project_to_color_depth(s["colour"], s["image"], s["view"])
    return [s["colour"], s["image"]]


# ---------------------------------------------------------------------------
# What a pass cannot do without.

def _seen(case, n):
    """Share of the volume inside the image per frame (mean), and inside any of the frames, on a coarse grid."""
    g, cam = _grid(case), CAMERAS[case["camera"]]
    ax = [(np.arange(16) + 0.5) / 16 * p + o for p, o in zip(g["physical_size"], g["global_offset"])]
    p = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    seen = []
    for q in _poses(case, 0, n):
        c = p @ S.matrix_from_quat(q[:4]).T + q[4:]
        with np.errstate(divide="ignore", invalid="ignore"):
            u, v = cam.fx * c[:, 0] / c[:, 2] + cam.cx, cam.fy * c[:, 1] / c[:, 2] + cam.cy
        seen.append((c[:, 2] > 0) & (u >= 0) & (u < cam.width) & (v >= 0) & (v < cam.height))
    seen = np.array(seen)
    return float(seen.mean()), float(seen.any(0).mean())


def work(case):
    kind, F = case["kind"], case["frames"]
    cam = CAMERAS[case["camera"]]
    pixels = cam.width * cam.height
    pix_bytes = 2 if case.get("depth") == "u16" else 4
    voxels = case["nx"] * case["ny"] * case["nz"] if "nx" in case else 0
    if kind == "live":   # the distances and weights of the voxels in view, read and written, and the frame
        each, _ = _seen(case, 8)
        return {"bytes": 16 * each * voxels + pixels * pix_bytes, "flops": 40 * each * voxels}
    if kind in ("sequence", "scan"):   # the finished volume written, the frames read, each frame's voxels updated
        each, _ = _seen(case, min(F, 16))
        return {"bytes": 8 * voxels + F * pixels * pix_bytes, "flops": 40 * each * voxels * F}
    if kind == "scenes":
        each, _ = _seen(case, 16)
        vf = [(int(np.prod(_scene_extents(case, k))), _scene_frames(case, k)) for k in range(case["scenes"])]
        return {"bytes": sum(8 * v + f * pixels * pix_bytes for v, f in vf),
                "flops": 40 * each * sum(v * f for v, f in vf)}
    if kind in ("mesh", "indexed"):   # distances and weights read, a surface of about 3 N^(2/3) triangles written
        tris = 3.0 * voxels ** (2.0 / 3.0)
        out = 48 * tris if kind == "mesh" else 12 * tris + 24 * tris / 2
        return {"bytes": 8 * voxels + out, "flops": 8 * voxels}
    if kind == "diff":   # volume, model, mask, result and the frames with their gradients, each once
        b = 8 if case["dtype"] == "f64" else 4
        each, _ = _seen(case, F)
        return {"bytes": b * (6 * voxels + 2 * F * pixels), "flops": 200 * each * voxels * F}
    points = F * pixels
    if kind == "cloud":
        return {"bytes": points * (pix_bytes + 33 + (3 if case["colour"] else 0)), "flops": 40 * points}
    return {"bytes": points * 33 + pixels * (4 + (3 if case["colour"] else 0)), "flops": 40 * points}


# ---------------------------------------------------------------------------
# The results in 64 bits, from the definitions.

def _depth64(d, scale=0.001):
    if d.dtype == torch.int16:
        return (d.to(torch.int32) & 0xFFFF).double() * float(np.float32(scale))
    return d.double()


def _axes64(g):
    out = []
    for n, p, o in zip(g["voxel_grid_size"], g["physical_size"], g["global_offset"]):
        vs = float(np.float32(p) / np.float32(n))
        out.append((torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * vs + float(np.float32(o)))
    return out


def _rotation64(q, mode):
    w, x, y, z = (float(v) for v in q)
    if mode == "fixed":
        n = math.sqrt(w * w + x * x + y * y + z * z)
        w, x, y, z = w / n, x / n, y / n, z / n
    else:
        w, x, y, z = (float(np.float32(v)) for v in (w, x, y, z))
    return [[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
            [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
            [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]


def _integrate64(case, depths, poses, extents=None):
    g, cam = _grid(case, extents), CAMERAS[case["camera"]]
    X, Y, Z = _axes64(g)
    vs = [float(np.float32(p) / np.float32(n)) for p, n in zip(g["physical_size"], g["voxel_grid_size"])]
    trunc = float(np.float32(1.1)) * math.sqrt(sum(v * v for v in vs))
    D = torch.full((len(Z), len(Y), len(X)), trunc, dtype=torch.float64, device=DEV)
    W = torch.zeros_like(D)
    step = max(1, (1 << 24) // (len(X) * len(Y)))
    fixed = case["mode"] == "fixed"
    f32 = [_depth64(d) for d in depths] if len(depths) <= 64 else None
    for z0 in range(0, len(Z), step):
        zz = Z[z0:z0 + step, None, None]
        d, w = D[z0:z0 + step], W[z0:z0 + step]
        for k in range(len(depths)):
            R = _rotation64(poses[k][:4], case["mode"])
            t = [float(v) if fixed else float(np.float32(v)) for v in poses[k][4:]]
            c = [r[0] * X[None, None, :] + (r[1] * Y[None, :, None] + (r[2] * zz + b)) for r, b in zip(R, t)]
            u, v = cam.fx * c[0] / c[2] + cam.cx, cam.fy * c[1] / c[2] + cam.cy
            if fixed:
                u, v = u.round_(), v.round_()
            else:
                u, v = u.trunc_(), v.trunc_()
                zero = (c[2] == 0) | (zz == 0)
                u.masked_fill_(zero, 0.0)
                v.masked_fill_(zero, 0.0)
            ok = (u >= 0) & (u < cam.width) & (v >= 0) & (v < cam.height)
            if fixed:
                ok &= c[2] > 0
            i = torch.where(ok, v * cam.width + u, torch.zeros_like(u)).long()
            dv = (f32[k] if f32 is not None else _depth64(depths[k])).reshape(-1)[i]
            sdf = dv - (c[2] if fixed else zz)
            ok &= (dv > 0) & (dv <= 24.0) & (sdf >= -trunc)
            tsdf = sdf.clamp_(max=trunc)
            if fixed:
                n = w.floor() + 1
                w.copy_(torch.where(ok, (w + 1).clamp_(max=128.0), w))
            else:
                n = w + 1
                w.copy_(torch.where(ok, n, w))
            d.copy_(torch.where(ok, d + (tsdf - d) / n, d))
    return D, W


# Cube corner k is at (x, y, z) + CORNERS[k]; edge e runs between corners EDGES[e]; TRIANGLES: for each of the 256
# sign patterns (bit k: corner k below zero) its triangles, three edges (hexadecimal) each: the classic
# Lorensen-Cline table in Cory Bloyd's public-domain layout.
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 0, 1), (0, 0, 1), (0, 1, 0), (1, 1, 0), (1, 1, 1), (0, 1, 1)]
EDGES = [(0, 1), (2, 1), (3, 2), (3, 0), (4, 5), (6, 5), (7, 6), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]
TRIANGLES = """
- 083 019 183981 12a 08312a 92a029 2832a8a98 3b2 0b28b0 19023b 1b219b98b 3a1ba3 0a108a8ba 3903b9ba9 98aa8b 478
430734 019847 419471731 12a847 34730412a 92a902847 2a9297273794 8473b2 b47b24204 90184723b 47b94b9b2921
3a13ba784 1ba14b1047b4 47890b9bab03 47b4b99ba 954 954083 054150 854835315 12a954 30812a495 52a542402
2a5325354348 95423b 0b208b495 05401523b 21525828b485 a3ba13954 4950818a18ba 54050b5bab03 54858aa8b 978579
930953573 078017157 153357 978957a12 a12950530573 802825857a52 2a5253357 7957893b2 95797292027b 23b018178157
b21b17715 958857a13a3b 5705097b010aba0 ba0b03a50807570 ba57b5 a65 0835a6 9015a6 1831985a6 165261 165126308
965906026 598582526328 23ba65 b08b20a65 01923b5a6 5a61929b298b 63b653513 08b0b50515b6 3b6036065059 65969bb98
5a6478 43047365a 1905a6847 a65197173794 612651478 125526304347 847905065026 739794329596269 3b2784a65
5a647242027b 01947823b5a6 9219b294b7b45a6 8473b53515b6 51b5b610b7b404b 059065036b63847 65969b4797b9 a4964a
4a649a083 a01a60640 83181686461a 149124264 308129249264 024426 832824426 a49a64b23 08228b49a4a6 3b201606461a
64161a48121b8b1 964936913b63 8b1810b61914641 3b6360064 648b68 7a678a89a 0730a709a67a a671a7178180 a67a71173
126168189867 269291679093739 780706602 732672 23ba68a89867 20727b09767a9a7 1801781a767a23b b21b17a61671
896867916b63136 091b67 7807063b0b60 7b6 76b 308b76 019b76 819831b76 a126b7 12a3086b7 2902a96b7 6b72a3a83a98
723627 708760620 276237019 162186198876 a76a17137 a7617a187108 03707a0a96a7 76a7a88a9 684b86 36b306046
86b846901 946963931b36 6846b82a1 12a30b06b046 4b846b0292a9 a93a32943b36463 823842462 042462 190234246438
194142246 8138618466a1 a10a06604 4634386a3039a93 a946a4 49576b 083495b76 50154076b b76834354315 954a1276b
6b712a083495 76b54a42a402 348354325a52b76 723762549 954086062687 362376150540 628687218485158 954a16176137
16a176107870954 40a4a503a6a737a 76a7a854a48a 6956b9b89 36b063056095 0b805b01556b 6b3635531 12a95b9b8b56
0b306b09656912a b85b56805a52025 6b36352a3a53 589528562382 956960062 158180568382628 156216 13616a386569896
a10a06950560 03856a a56 b5a75b b5ab75830 5b75ab190 a75ab7981831 b12b71751 08312717572b 9759279022b7
75272b592328982 25a235375 820852875a25 9015a35373a2 982921872a25752 135375 087071175 903935537 987597
5845a8ab8 5045b05abb30 01984a8aba45 ab4a45b34941314 2512852b8458 04b0b345b2b151b 0250592b5458b85 9452b3
25a352345384 5a2524420 3a235a385458019 5a2524192942 845853351 045105 845853905035 945 4b749b9ab 0834979b79ab
1ab1b414074b 3143481a474bab4 4b79b492b912 9749b791b2b1083 b74b42240 b74b42834324 29a279237749 9a7974a27870207
37a3a274a1a040a 1a2874 491417713 491417081871 403743 487 9a8ab8 30939bb9a 01a0a88ab 31ab3a 12b1b99b8
30939b1292b9 02b80b 32b 23828aa89 9a2092 23828a0181a8 1a2 138918 091 038 -
""".split()


def _lower_first(e):
    a, b = EDGES[e]
    return (a, b) if sum(CORNERS[a]) < sum(CORNERS[b]) else (b, a)


def _cubes64(case, vol):
    """Distances in 64 bits, and per cube (linear order) whether it is meshed and its sign pattern.  The compat mode
    reads layers nx + ny voxels apart, as the reference does, and does not ask whether voxels were observed."""
    D, W = vol.voxel_distances_data().double(), vol.voxel_weights_data()
    nz, ny, nx = D.shape
    pat = torch.zeros((nz - 1, ny - 1, nx - 1), dtype=torch.int16, device=DEV)
    obs = torch.ones_like(pat, dtype=torch.bool)
    layer = nx + ny if case["mode"] == "compat" else nx * ny
    for k, (dx, dy, dz) in enumerate(CORNERS):
        def at(v):
            return v.as_strided(pat.shape, (layer, nx, 1), dz * layer + dy * nx + dx)
        pat |= (at(D) < 0).to(torch.int16) << k
        if case["mode"] == "fixed":
            obs &= at(W) > 0
    return D, pat, obs


def _edge_points64(D, g, lo, hi):
    """Points where the surface crosses between voxels lo and hi (linear numbers), and how far along."""
    nz, ny, nx = D.shape
    ax = _axes64(g)
    sa, sb = D.reshape(-1)[lo], D.reshape(-1)[hi]
    r = (sa / (sa - sb))[:, None]
    pa, pb = (torch.stack([ax[0][v % nx], ax[1][v // nx % ny], ax[2][v // (nx * ny)]], -1) for v in (lo, hi))
    return pa + r * (pb - pa), r


def _mesh64(case, vol):
    D, pat, obs = _cubes64(case, vol)
    pat = torch.where(obs, pat, torch.zeros_like(pat))
    count = torch.tensor([0 if w == "-" else len(w) // 3 for w in TRIANGLES], device=DEV)
    edge = torch.zeros((256, 5, 3), dtype=torch.long)
    for p, w in enumerate(TRIANGLES):
        for k, ch in enumerate(w if w != "-" else ""):
            edge[p, k // 3, k % 3] = int(ch, 16)
    ends = torch.tensor([[CORNERS[k] for k in _lower_first(e)] for e in range(12)], device=DEV)
    z, y, x = torch.nonzero((pat > 0) & (pat < 255), as_tuple=True)
    p = pat[z, y, x].long()
    at = torch.repeat_interleave(torch.arange(len(p), device=DEV), count[p])
    first = torch.cumsum(count[p], 0) - count[p]
    e = edge.to(DEV)[p[at], torch.arange(len(at), device=DEV) - first[at]].reshape(-1)
    nz, ny, nx = D.shape
    layer = nx + ny if case["mode"] == "compat" else nx * ny
    base = (z * layer + y * nx + x)[at].repeat_interleave(3, 0)
    lo, hi = (base + (ends[e, k] * torch.tensor([1, nx, layer], device=DEV)).sum(-1) for k in (0, 1))
    return _edge_points64(D, _grid(case), lo, hi)[0].reshape(-1, 3, 3)


def _indexed64(case, vol):
    D, pat, obs = _cubes64(case, vol)
    nz, ny, nx = D.shape
    used = torch.zeros((nz, ny, nx, 3), dtype=torch.bool, device=DEV)
    for e in range(12):
        a, b = _lower_first(e)
        (dx, dy, dz), q = CORNERS[a], [i for i in range(3) if CORNERS[a][i] != CORNERS[b][i]][0]
        crossed = obs & (((pat >> a) ^ (pat >> b)) & 1).bool()
        used[dz:nz - 1 + dz, dy:ny - 1 + dy, dx:nx - 1 + dx, q] |= crossed
    z, y, x, q = torch.nonzero(used, as_tuple=True)
    lo = torch.stack([x, y, z], -1)
    hi = lo + torch.nn.functional.one_hot(q, 3)
    flat = torch.tensor([1, nx, nx * ny], device=DEV)
    pts, r = _edge_points64(D, _grid(case), (lo * flat).sum(-1), (hi * flat).sum(-1))
    vs = [float(a[1] - a[0]) for a in _axes64(_grid(case))]

    def gradient(v):
        out = []
        for i, n in enumerate((nx, ny, nz)):
            up, dn = v.clone(), v.clone()
            up[:, i] = (v[:, i] + 1).clamp(max=n - 1)
            dn[:, i] = (v[:, i] - 1).clamp(min=0)
            diff = D[up[:, 2], up[:, 1], up[:, 0]] - D[dn[:, 2], dn[:, 1], dn[:, 0]]
            out.append(diff / ((up[:, i] - dn[:, i]).double() * vs[i]))
        return torch.stack(out, -1)

    ga, gb = gradient(lo), gradient(hi)
    n = ga + r * (gb - ga)
    return pts, torch.nn.functional.normalize(n, dim=-1, eps=1e-300)


def _diff64(case, s):
    cfg, cam = s["cfg"], CAMERAS[case["camera"]]
    depth = s["depth"].detach().double().requires_grad_(True)
    R = s["R"].detach().double().requires_grad_(True)
    t = s["t"].detach().double().requires_grad_(True)
    x, y, z = _axes64(_grid(case))
    D, W = s["D0"].double(), s["W0"].double()
    tr = float(np.float32(cfg.truncation))
    for f in range(case["frames"]):
        c = [R[f, k, 0] * x[None, None, :] + R[f, k, 1] * y[None, :, None] + R[f, k, 2] * z[:, None, None] + t[f, k]
             for k in range(3)]
        front = c[2] > float(np.float32(cfg.min_z))
        cz = torch.where(front, c[2], torch.ones_like(c[2]))
        u, v = cam.fx * c[0] / cz + cam.cx, cam.fy * c[1] / cz + cam.cy
        ok = front & (u > -1) & (v > -1) & (u < cam.width) & (v < cam.height)
        u, v = torch.where(ok, u, torch.zeros_like(u)), torch.where(ok, v, torch.zeros_like(v))
        fu, fv = u.detach().floor(), v.detach().floor()
        a, b = u - fu, v - fv
        wv = torch.zeros_like(u)
        nd = torch.zeros_like(u)
        flat = depth[f].reshape(-1)
        for k, bw in enumerate(((1 - a) * (1 - b), a * (1 - b), (1 - a) * b, a * b)):
            px, py = fu.long() + (k & 1), fv.long() + (k >> 1)
            inside = (px >= 0) & (py >= 0) & (px < cam.width) & (py < cam.height)
            dv = flat[torch.where(inside, py * cam.width + px, torch.zeros_like(px))]
            valid = inside & (dv > 0) & (dv <= cfg.max_depth)
            wv = wv + torch.where(valid, bw, torch.zeros_like(bw))
            nd = nd + torch.where(valid, bw * dv, torch.zeros_like(bw))
        ok = ok & (wv > 0)
        sdf = nd / torch.where(ok, wv, torch.ones_like(wv)) - c[2]
        tsdf = torch.where(sdf > tr, torch.full_like(sdf, tr), sdf)
        band = (sdf + tr) * (2.0 / tr)
        band = torch.where(band >= 1, torch.ones_like(band), torch.where(band > 0, band, torch.zeros_like(band)))
        w = torch.where(ok, wv * band, torch.zeros_like(wv))
        ok = w > 0
        sw = torch.where(ok, W + w, torch.ones_like(W))
        D = torch.where(ok, D + w * (tsdf - D) / sw, D)
        W = torch.where(ok, torch.where(sw < cfg.max_weight, sw, torch.full_like(sw, cfg.max_weight)), W)
    cw = s["mask"].double() * W
    loss = (cw * (D - s["model"].double()) ** 2).sum() / cw.sum()
    g = torch.autograd.grad(loss, (depth, R, t))
    return [D.detach(), W.detach(), loss.detach()] + list(g)


def _project64(case, s):
    """The z-buffer's depth image: per pixel the smallest camera z of the points that fall on it, 0 where none."""
    cam = CAMERAS[case["camera"]]
    p = s["pc"].get_points()[:, :12].contiguous().view(torch.float32).double()
    R, t = _rotation64(s["view"][:4], "compat"), [float(np.float32(v)) for v in s["view"][4:]]
    c = [r[0] * p[:, 0] + r[1] * p[:, 1] + r[2] * p[:, 2] + b for r, b in zip(R, t)]
    u, v = (c[0] * cam.fx / c[2] + cam.cx).trunc(), (c[1] * cam.fy / c[2] + cam.cy).trunc()
    ok = (c[2] != 0) & (u >= 0) & (u < cam.width) & (v >= 0) & (v < cam.height)
    i = (v[ok] * cam.width + u[ok]).long()
    z = torch.full((cam.height * cam.width,), math.inf, dtype=torch.float64, device=DEV)
    z.scatter_reduce_(0, i, c[2][ok], "amin")
    return torch.where(torch.isinf(z), torch.zeros_like(z), z).reshape(cam.height, cam.width)


def exact(case, seed):
    kind = case["kind"]
    if kind == "scenes":
        out = []
        for k in range(case["scenes"]):
            d, p = _frames(case, int(seed) * 16 + k, _scene_frames(case, k))
            out += list(_integrate64(case, d, p, _scene_extents(case, k)))
        return out
    if kind in ("live", "sequence", "scan"):
        d, p = _frames(case, int(seed), 8 if kind == "live" else case["frames"])
        n = 1 if kind == "live" else len(d)
        return list(_integrate64(case, d[:n], p[:n]))
    if kind == "cloud":
        return None   # packed records: bytes
    s = prepare(case, seed)
    if kind == "mesh":
        return [_mesh64(case, s["vol"]), None]
    if kind == "indexed":
        return list(_indexed64(case, s["vol"])) + [None]
    if kind == "diff":
        return _diff64(case, s)
    image = _project64(case, s)
    return [image] if s["colour"] is None else [None, image]
