"""Timed cases of the reconstruction path, each through its public entry points.

Every case works on a seeded synthetic room that is rendered on the GPU: walls
of a 4 x 4 x 3 m room with spheres and boxes along them, seen by a hand-held
camera that moves at most 6 mm and 0.6 degrees a frame, as uint16 millimetre
depth with a depth sensor's noise (sigma 1.2 mm + 1.9 mm (z - 0.4)^2) and 5 %
of the pixels missing. The kinds of work are

* ``preprocess``  a frame's point cloud and normals (depth_to_pcd, normals_from_pcd);
* ``dropin``      one frame of the reference's call surface: integrate with
                  colour, raycast, kokkos_icp against the frame before;
* ``keyframe``    a sliding window of fused frames: integrate the new one,
                  deIntegrate the oldest, raycast the view;
* ``track``       one frame of the per-frame pipeline: upload from pinned host
                  memory, track, integrate, raycast the model view, read the pose;
* ``icp``         kokkos_icp between two frames with a perturbed start;
* ``refuse``      loop-closure re-fusion of a batch of keyframes, then the model
                  view of the corrected volume;
* ``loss``        the differentiable raycast's loss and its pose gradient, with
                  the voxel gradients where ``voxels`` is set;
* ``mesh``        marching cubes of the whole volume.

A pass on the fused volume returns what the caller gets back from it, a view
of the volume (point, colour and normal maps, poses, triangles); the volume
itself stays in the grid, as it does in use. Views, tracked poses, losses of a
volume and meshes follow decisions that single-precision roundings make (which
pixel a voxel projects to, which voxel a ray crosses in), so they have no
value in 64 bits of their own; point clouds, normals and the pose of an ICP
alignment have, and exact() computes them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from superscanner_gb300 import GPUVoxelGrid, depth_to_pcd, kokkos_icp, normals_from_pcd
from superscanner_gb300.mesh import extract_triangles
from superscanner_gb300.pipeline import FORMS, Pipeline, raycast_maps
from superscanner_gb300.raydiff import raycast_loss_grad

ROOM = (4.0, 4.0, 3.0)
MAX_WEIGHT = 255.0


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest call: a quarter-size frame turned into points and normals for a registration front end
        dict(name="preprocess_qvga", kind="preprocess", rows=240, cols=320),
        # the reference's frame loop on a coarse preview volume, where launches and host work count
        dict(name="dropin_preview", kind="dropin", rows=120, cols=160, vl=0.008, buckets=1 << 16, storage="f32",
             color=True, plane=False),
        # the reference's frame loop at a depth camera's full size, with colour, over a window of frames
        dict(name="keyframe_vga_color", kind="keyframe", rows=480, cols=640, vl=0.004, buckets=1 << 19, storage="f32",
             color=True, window=6),
        # a cropped (odd) sensor image, half-precision volume, no colour
        dict(name="keyframe_odd_f16", kind="keyframe", rows=389, cols=517, vl=0.005, buckets=1 << 18, storage="f16",
             color=False, window=6),
        # a preview of the tracker: latency of one frame
        dict(name="track_preview", kind="track", rows=120, cols=160, vl=0.008, buckets=1 << 16, form="chosen",
             margin=0.04),
        # the headline workload: 640 x 480 at 4 mm
        dict(name="track_vga", kind="track", rows=480, cols=640, vl=0.004, buckets=1 << 20, form="chosen",
             margin=0.04),
        # a 720p depth camera
        dict(name="track_hd", kind="track", rows=720, cols=1280, vl=0.004, buckets=1 << 20, form="chosen",
             margin=0.04),
        # frame-to-frame registration, point to plane, full size
        dict(name="icp_vga_plane", kind="icp", rows=480, cols=640, plane=True),
        # loop closure: 200 keyframes whose poses a pose graph corrected by up to 2 degrees and 3 cm
        dict(name="refuse_vga_200", kind="refuse", rows=480, cols=640, vl=0.004, buckets=1 << 20, frames=200,
             exact_fusion=False),
        # pose refinement by gradient: one evaluation at full size
        dict(name="loss_pose_vga", kind="loss", rows=480, cols=640, vl=0.004, buckets=1 << 18, voxels=False),
        # map refinement by gradient: pose and voxel gradients, odd size
        dict(name="loss_voxels_odd", kind="loss", rows=389, cols=517, vl=0.006, buckets=1 << 15, voxels=True),
        # the end of a scan: the mesh of a room
        dict(name="mesh_room", kind="mesh", rows=480, cols=640, vl=0.004, buckets=1 << 20, storage="f16", frames=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["preprocess", "dropin", "keyframe", "track", "icp", "refuse", "loss", "mesh"])
    top = {"preprocess": 720, "dropin": 600, "keyframe": 600, "track": 720, "icp": 600, "refuse": 480, "loss": 600,
           "mesh": 480}[kind]
    rows = _log_int(rng, 90, top)
    cols = int(rows * rng.uniform(1.2, 1.78))
    c = dict(kind=kind, rows=rows, cols=cols)
    if kind in ("preprocess",):
        return c
    if kind == "icp":
        return dict(c, plane=rng.random() < 0.5)
    vl = round(rng.uniform(0.004, 0.01), 4)
    c.update(vl=vl, buckets=1 << (20 if vl < 0.005 else 19 if vl < 0.0065 else 18))
    storage = rng.choice(["f32", "f16"])
    if kind == "dropin":
        return dict(c, storage=storage, color=rng.random() < 0.7, plane=rng.random() < 0.5)
    if kind == "keyframe":
        return dict(c, storage=storage, color=rng.random() < 0.5, window=rng.randint(2, 8))
    if kind == "track":
        return dict(c, form=rng.choice(["chosen", "chosen", "plain"]), margin=0.04 if vl < 0.008 else 5 * vl)
    if kind == "refuse":
        return dict(c, frames=_log_int(rng, 4, 200), exact_fusion=rng.random() < 0.3)
    if kind == "loss":
        c["buckets"] = 1 << (17 if vl < 0.005 else 16)
        return dict(c, voxels=rng.random() < 0.4)
    return dict(c, storage=storage, frames=rng.randint(6, 24))


# ----------------------------------------------------------------- the scene

def _intrinsic(case):
    f = 525.0 * case["cols"] / 640.0
    return f, f, (case["cols"] - 1) / 2.0, (case["rows"] - 1) / 2.0


def _trajectory(g, n, step):
    """n camera -> world poses along a ring around the room's centre, looking outwards and down."""
    phase, tilt = g.uniform(0, 2 * math.pi), g.uniform(-4.0, 4.0)
    out = np.zeros((n, 4, 4))
    for k in range(n):
        t = k * step
        w = 2 * math.pi / 500.0 * t + phase
        yaw = phase + math.radians(0.6) * t
        pitch = math.radians(-25.0 + tilt + 8.0 * math.sin(1.7 * w))
        z = np.array([math.cos(yaw) * math.cos(pitch), math.sin(yaw) * math.cos(pitch), math.sin(pitch)])
        x = np.cross(z, [0.0, 0.0, 1.0])
        x /= np.linalg.norm(x)
        out[k, :3, :3] = np.stack([x, np.cross(z, x), z], axis=1)
        out[k, :3, 3] = [0.64 * math.cos(w), 0.5 * math.sin(w), 0.9 + 0.12 * math.sin(2.3 * w)]
        out[k, 3, 3] = 1.0
    return out


def _objects(g):
    """(spheres [n, 4], boxes [m, 6]) along the walls of the room, clear of the camera's ring."""
    lim = np.array([ROOM[0] / 2, ROOM[1] / 2])
    spheres, boxes = [], []
    for k in range(14):
        r = g.uniform(0.1, 0.4)
        c = g.uniform(-1.0, 1.0, 2) * (lim - r - 0.05)
        ax = k % 2
        c[ax] = (1 if (k // 2) % 2 else -1) * (lim[ax] - r - g.uniform(0.0, 0.35))
        spheres.append([c[0], c[1], r if k % 3 else g.uniform(r, 2.0), r])
    for k in range(10):
        h = g.uniform(0.08, 0.3, 3)
        c = g.uniform(-1.0, 1.0, 2) * (lim - h[:2] - 0.05)
        ax = k % 2
        c[ax] = (1 if (k // 2) % 2 else -1) * (lim[ax] - h[ax])
        boxes.append([c[0] - h[0], c[1] - h[1], 0.0, c[0] + h[0], c[1] + h[1], 2 * h[2]])
    return np.array(spheres), np.array(boxes)


def _render(case, poses, objects, seed, color):
    """Depth [n, rows, cols] (int16 view of uint16 millimetres) and colour [n, rows, cols, 3] uint8, on the GPU."""
    rows, cols = case["rows"], case["cols"]
    fx, fy, cx, cy = _intrinsic(case)
    dev = "cuda"
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    j = (torch.arange(cols, device=dev, dtype=torch.float32) - cx) / fx
    i = (torch.arange(rows, device=dev, dtype=torch.float32) - (rows - cy)) / fy
    depth = torch.empty((len(poses), rows, cols), dtype=torch.int16, device=dev)
    rgb = torch.empty((len(poses), rows, cols, 3), dtype=torch.uint8, device=dev) if color else None
    chunk = max(1, 8_000_000 // (rows * cols))
    spheres, boxes = objects
    for a in range(0, len(poses), chunk):
        T = torch.as_tensor(poses[a:a + chunk], dtype=torch.float32, device=dev)
        n = len(T)
        o = [T[:, k, 3].view(n, 1, 1) for k in range(3)]
        d = [T[:, k, 0].view(n, 1, 1) * j.view(1, 1, -1) + T[:, k, 1].view(n, 1, 1) * i.view(1, -1, 1)
             + T[:, k, 2].view(n, 1, 1) for k in range(3)]
        inv = [1.0 / torch.where(v.abs() < 1e-7, torch.full_like(v, 1e-7), v) for v in d]
        lo, hi = (-ROOM[0] / 2, -ROOM[1] / 2, 0.0), (ROOM[0] / 2, ROOM[1] / 2, ROOM[2])
        t = torch.full_like(d[0], 1e9)
        for k in range(3):
            t = torch.minimum(t, torch.maximum((lo[k] - o[k]) * inv[k], (hi[k] - o[k]) * inv[k]))
        dd = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        for s in spheres.tolist():
            oc = [o[k] - s[k] for k in range(3)]
            b = oc[0] * d[0] + oc[1] * d[1] + oc[2] * d[2]
            c = oc[0] * oc[0] + oc[1] * oc[1] + oc[2] * oc[2] - s[3] * s[3]
            disc = b * b - dd * c
            hit = (-b - disc.clamp_min(0.0).sqrt()) / dd
            t = torch.where((disc > 0) & (hit > 1e-3) & (hit < t), hit, t)
        for s in boxes.tolist():
            near, far = torch.full_like(t, -1e9), torch.full_like(t, 1e9)
            for k in range(3):
                u, v = (s[k] - o[k]) * inv[k], (s[3 + k] - o[k]) * inv[k]
                near, far = torch.maximum(near, torch.minimum(u, v)), torch.minimum(far, torch.maximum(u, v))
            t = torch.where((near < far) & (near > 1e-3) & (near < t), near, t)
        if color:
            p = [o[k] + t * d[k] for k in range(3)]
            check = ((p[0] * 10).floor() + (p[1] * 10).floor() + (p[2] * 10).floor()) % 2
            for k in range(3):
                rgb[a:a + n, ..., k] = ((90 + 50 * torch.sin(1.5 * p[k] + k) + 60 * check).clamp(0, 255)).to(torch.uint8)
        t = t + (0.0012 + 0.0019 * (t - 0.4) ** 2) * torch.randn(t.shape, device=dev, generator=gen)
        keep = torch.rand(t.shape, device=dev, generator=gen) >= 0.05
        depth[a:a + n] = torch.where(keep, (t * 1000.0 + 0.5).floor().clamp(0, 32767), torch.zeros_like(t)).to(torch.int16)
    return depth, rgb


def _small_motion(g, degrees, metres):
    """A rigid motion of up to so many degrees and metres."""
    ax = g.normal(size=3)
    ax /= np.linalg.norm(ax)
    a = math.radians(g.uniform(0.2, 1.0) * degrees)
    K = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
    T = np.eye(4)
    T[:3, :3] += math.sin(a) * K + (1 - math.cos(a)) * K @ K
    v = g.normal(size=3)
    T[:3, 3] = v / np.linalg.norm(v) * g.uniform(0.2, 1.0) * metres
    return T


def _sequence(case, seed, n, step=1.0, color=False):
    """(poses, depth, rgb, the seed's generator)."""
    g = np.random.default_rng(seed)
    objects = _objects(g)
    poses = _trajectory(g, n, step)
    depth, rgb = _render(case, poses, objects, seed, color)
    return poses, depth, rgb, g


def _icp_pair(case, seed):
    poses, depth, _, g = _sequence(case, seed, 5)
    return depth[4], depth[0], _small_motion(g, 0.5, 0.005) @ poses[4], poses[0]


def _grid(case, storage, color, max_weight=0.0):
    vl = case["vl"]
    g = GPUVoxelGrid(int(1e9), 4 * vl, vl, case["rows"], case["cols"], storage=storage, with_color=color,
                     hash_buckets=case["buckets"], max_weight=max_weight)
    g.setIntrinsic(*_intrinsic(case))
    return g


class _Buffer:
    """A device buffer of a pipeline, as torch takes it without a copy; a tensor of it keeps the pipeline."""

    def __init__(self, pipe, ptr, shape):
        self.pipe = pipe
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False), version=3)


# ------------------------------------------------------------------- prepare

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, at=0)
    if kind == "preprocess":
        _, depth, _, _ = _sequence(case, seed, 1)
        return dict(s, depth=depth[0], intr=_intrinsic(case))
    if kind == "icp":
        d1, d2, tx, ty = _icp_pair(case, seed)
        return dict(s, d1=d1, d2=d2, tx=tx, ty=ty, intr=_intrinsic(case))
    if kind == "dropin":
        poses, depth, rgb, g = _sequence(case, seed, 6, color=case["color"])
        start = [_small_motion(g, 0.5, 0.005) @ T for T in poses]
        grid = _grid(case, case["storage"], case["color"])
        grid.integrate(rgb[0] if case["color"] else None, depth[0], poses[0], case["color"])
        return dict(s, grid=grid, poses=poses, start=start, depth=depth, rgb=rgb, intr=_intrinsic(case))
    if kind == "keyframe":
        n = 2 * case["window"]
        poses, depth, rgb, _ = _sequence(case, seed, n, color=case["color"])
        grid = _grid(case, case["storage"], case["color"])
        for k in range(case["window"]):
            grid.integrate(rgb[k] if case["color"] else None, depth[k], poses[k], case["color"])
        return dict(s, grid=grid, poses=poses, depth=depth, rgb=rgb)
    if kind == "track":
        n = 8
        poses, depth, _, _ = _sequence(case, seed, n)
        form = FORMS[case["form"]]
        grid = _grid(case, form["storage"], False, MAX_WEIGHT)
        pipe = Pipeline(grid, use_graph=form["use_graph"], persistent_track=form["persistent_track"],
                        hint_margin=case["margin"])
        pipe.set_pose(poses[0])
        pipe.frame(depth[0], track=False)
        host = depth.cpu().pin_memory()
        shape = (case["rows"], case["cols"], 4)
        maps = [torch.as_tensor(_Buffer(pipe, p, shape), device="cuda") for p in pipe.maps()]
        pose = torch.zeros((4, 4), dtype=torch.float64).pin_memory()
        return dict(s, grid=grid, pipe=pipe, host=host, maps=maps, pose=pose,
                    order=list(range(1, n)) + list(range(n - 2, -1, -1)))
    if kind == "refuse":
        n = case["frames"]
        poses, depth, _, g = _sequence(case, seed, n, step=400.0 / max(n, 200))
        for k in range(n):  # something close to the camera hides a part of the view
            h, w = (int(v * math.sqrt(g.uniform(0.0, 0.6))) for v in (case["rows"], case["cols"]))
            r, c = int(g.integers(0, case["rows"] - h)), int(g.integers(0, case["cols"] - w))
            depth[k, r:r + h, c:c + w] = 0
        grid = _grid(case, "f16", False, MAX_WEIGHT)
        for k in range(n):
            grid.integrate_fast(depth[k], poses[k])
        new = np.stack([_small_motion(g, 2.0, 0.03) @ T for T in poses])
        grid.refuse_batch([], [], [])
        return dict(s, grid=grid, depth=list(depth), poses=[poses, new])
    if kind == "loss":
        poses, depth, _, g = _sequence(case, seed, 6)
        grid = _grid(case, "f16", False, MAX_WEIGHT)
        for k in range(6):
            grid.integrate_fast(depth[k], poses[k])
        s.update(grid=grid, depth=depth[3], T=_small_motion(g, 1.0, 0.01) @ poses[3])
        if case["voxels"]:
            # voxel gradients come in the table's layout: rows of the blocks in key order, then rows of free buckets
            s["grad"] = torch.zeros((case["buckets"], 512), dtype=torch.float32, device="cuda")
            used = grid.export_buckets()
            free = np.setdiff1d(np.arange(case["buckets"]), used)
            s["order"] = torch.from_numpy(np.concatenate([used, free])[:case["buckets"] // 2]).cuda().long()
        return s
    poses, depth, _, _ = _sequence(case, seed, case["frames"], step=600.0 / case["frames"])
    grid = _grid(case, case["storage"], False, MAX_WEIGHT)
    for k in range(case["frames"]):
        grid.integrate_fast(depth[k], poses[k])
    room = int(160.0 / case["vl"] ** 2)
    weights = torch.linspace(1.0, 2.0, 9, dtype=torch.float64).sqrt().cuda()
    return dict(s, grid=grid, mesh=torch.zeros((room, 3, 3), device="cuda"), weights=weights)


# ----------------------------------------------------------------------- run

def run(s):
    case, at = s["case"], s["at"]
    s["at"] += 1
    kind = case["kind"]
    if kind == "preprocess":
        pcd = depth_to_pcd(s["depth"], *s["intr"])
        return dict(pcd=pcd, normals=normals_from_pcd(pcd))
    if kind == "icp":
        T, rmse = kokkos_icp(s["d1"], s["d2"], s["tx"], s["ty"], int(case["plane"]), s["intr"])
        return dict(T=T, rmse=rmse)
    grid = s.get("grid")
    if kind == "dropin":
        n = len(s["poses"])
        last, k = at % n, (at + 1) % n
        color = case["color"]
        grid.integrate(s["rgb"][k] if color else None, s["depth"][k], s["poses"][k], color)
        pcd, col = grid.raycast(s["poses"][k], with_color=color)
        T, rmse = kokkos_icp(s["depth"][k], s["depth"][last], s["start"][k], s["poses"][last], int(case["plane"]),
                             s["intr"])
        return dict(pcd=pcd, color=col, T=T, rmse=rmse) if color else dict(pcd=pcd, T=T, rmse=rmse)
    if kind == "keyframe":
        n, w, color = len(s["poses"]), case["window"], case["color"]
        new, old = (at + w) % n, at % n
        rgb = s["rgb"]
        grid.integrate(rgb[new] if color else None, s["depth"][new], s["poses"][new], color)
        grid.deIntegrate(rgb[old] if color else None, s["depth"][old], s["poses"][old], color)
        pcd, col = grid.raycast(s["poses"][new], with_color=color)
        return dict(pcd=pcd, color=col) if color else dict(pcd=pcd)
    if kind == "track":
        k = s["order"][at % len(s["order"])]
        s["pipe"].frame(s["host"][k])
        s["pipe"].read_pose_async(s["pose"].data_ptr())
        return dict(pose=s["pose"], vertex_depth=s["maps"][0], normal=s["maps"][1])
    if kind == "refuse":
        old, new = s["poses"] if at % 2 == 0 else s["poses"][::-1]
        grid.refuse_batch(s["depth"], old, new, exact=case["exact_fusion"])
        vertex, normal = raycast_maps(grid, new[-1])
        return dict(vertex_depth=vertex, normal=normal)
    if kind == "loss":
        if case["voxels"]:
            s["grad"].zero_()
            loss, grad, valid = raycast_loss_grad(grid, s["T"], s["depth"], grad_voxels=s["grad"])
            return dict(loss=loss, grad=grad, valid=valid, voxels=s["grad"][s["order"]])
        loss, grad, valid = raycast_loss_grad(grid, s["T"], s["depth"])
        return dict(loss=loss, grad=grad, valid=valid)
    # the soup comes in no fixed order: put in one, into the caller's buffer, as one that compares or caches meshes does
    tris = extract_triangles(grid)
    n = len(tris)
    order = torch.argsort(torch.mv(tris.view(-1, 9).double(), s["weights"]))
    torch.index_select(tris, 0, order, out=s["mesh"][:n])
    s["mesh"][n:].zero_()
    return dict(triangles=s["mesh"], count=n)


# ---------------------------------------------------------------------- work

def work(case):
    kind, px = case["kind"], case["rows"] * case["cols"]
    if kind == "preprocess":
        return dict(bytes=px * (2 + 12 + 12), flops=px * 60)
    # ICP: both images in; 10 iterations of a 100-tap search (a distance each)
    icp = dict(bytes=px * 4 + 132, flops=px * 10 * 100 * 8)
    if kind == "icp":
        return icp
    vl, trunc = case["vl"], 4 * case["vl"]
    # a view sees about 5 m^2 of surface (scaled by its aspect); a band of +- trunc around it is fused
    area = 6.0 * case["rows"] / case["cols"] * 4 / 3
    band = area * 2 * trunc / vl ** 3
    fuse_flops = 40 * band
    if kind in ("dropin", "keyframe"):
        size = (8 if case["storage"] == "f32" else 4) + (12 if case["color"] else 0)
        frame = 2 + (3 if case["color"] else 0)
        view = dict(bytes=px * (12 + (12 if case["color"] else 0)) + area / vl ** 2 * size, flops=px * 60 * 20)
        times = 1 if kind == "dropin" else 2
        b = times * (px * frame + 2 * size * band) + view["bytes"]
        f = times * fuse_flops + view["flops"]
        return dict(bytes=b + icp["bytes"], flops=f + icp["flops"]) if kind == "dropin" else dict(bytes=b, flops=f)
    if kind == "track":
        size = 8 if case["form"] == "plain" else 4
        pixels = px * (10 + 5 / 4 + 4 / 16)
        return dict(bytes=px * (2 + 32 + 32) + 2 * size * band, flops=pixels * 120 + fuse_flops + px * 300)
    if kind == "refuse":
        return dict(bytes=case["frames"] * px * 2 + 2 * 4 * 6 * band + px * 32,
                    flops=case["frames"] * 2 * fuse_flops + px * 300)
    if kind == "loss":
        read = px * 2 + 4 * area / vl ** 2 * 2
        return dict(bytes=read + (2 * 4 * area / vl ** 2 * 2 if case["voxels"] else 0), flops=px * 600)
    surface = min(60.0, case["frames"] * 3.0)
    return dict(bytes=4 * surface * 2 * trunc / vl ** 3 + surface / vl ** 2 * 2 * 36,
                flops=surface * 2 * trunc / vl ** 3 * 20)


# --------------------------------------------------------------------- exact

def _points(case, depth):
    fx, fy, cx, cy = _intrinsic(case)
    rows, cols = case["rows"], case["cols"]
    d = depth.double() / 1000.0
    j = (torch.arange(cols, device=depth.device, dtype=torch.float64) - cx) / fx
    i = (torch.arange(rows, device=depth.device, dtype=torch.float64) - (rows - cy)) / fy
    return torch.stack([j.view(1, -1) * d, i.view(-1, 1) * d, d], dim=-1)


def _normals(p):
    out = torch.zeros_like(p)
    out[..., 2] = 1.0
    c, dn, up = p[1:-1, 1:-1], p[2:, 1:-1], p[:-2, 1:-1]
    rt, lf = p[1:-1, 2:], p[1:-1, :-2]
    cr = torch.linalg.cross
    n = cr(dn - c, rt - c) + cr(lf - c, dn - c) + cr(rt - c, up - c) + cr(up - c, lf - c)
    ok = (c[..., 2] != 0) & (dn[..., 2] != 0) & (up[..., 2] != 0) & (rt[..., 2] != 0) & (lf[..., 2] != 0)
    n = n / n.norm(dim=-1, keepdim=True)
    out[1:-1, 1:-1] = torch.where(ok[..., None], n, out[1:-1, 1:-1])
    return out


def _icp(case, d1, d2, tx, ty, plane):
    """The alignment in 64 bits: 10 iterations of the 10 x 10 window's nearest point (or tangent plane) within
    75 mm, the rigid motion of each from the SVD of the centred correlation, the one of the lowest RMSE kept."""
    fx, fy, cx, cy = _intrinsic(case)
    rows, cols = case["rows"], case["cols"]
    x, y = _points(case, d1).view(-1, 3), _points(case, d2)
    nrm = _normals(y).view(-1, 3)
    y = y.view(-1, 3)
    x = x[x[:, 2] != 0]
    T = torch.as_tensor(np.linalg.inv(ty) @ tx, device=x.device)
    best, lowest = torch.eye(4, dtype=torch.float64), math.inf
    for _ in range(10):
        px = x @ T[:3, :3].T + T[:3, 3]
        ci = (px[:, 1] * fy / px[:, 2] + (rows - cy)).trunc().long()
        cj = (px[:, 0] * fx / px[:, 2] + cx).trunc().long()
        inside = (ci > 5) & (ci < rows - 5) & (cj > 5) & (cj < cols - 5)
        xs, ps, ci, cj = x[inside], px[inside], ci[inside], cj[inside]
        small = torch.full((len(xs),), math.inf, dtype=torch.float64, device=x.device)
        found = torch.zeros_like(xs)
        for k in range(-5, 5):
            for l in range(-5, 5):
                q = (ci + k) * cols + cj + l
                t, n = y[q], nrm[q]
                if plane:
                    dist = ((t - ps) * n).sum(-1)
                    to, far, ok = ps + dist[:, None] * n, dist.abs(), (t[:, 2] != 0) & (n[:, 0] != 0)
                else:
                    to, far, ok = t, (t - ps).norm(dim=-1), t[:, 2] != 0
                ok &= (far < small) & (far < 0.075)
                small = torch.where(ok, far, small)
                found = torch.where(ok[:, None], to, found)
        ok = found[:, 2] != 0
        a, b = xs[ok], found[ok]
        rmse = float((b - a @ T[:3, :3].T - T[:3, 3]).square().sum(-1).mean().sqrt())
        ca, cb = a.mean(0), b.mean(0)
        U, _, Vh = torch.linalg.svd((a - ca).T @ (b - cb))
        T = torch.eye(4, dtype=torch.float64, device=x.device)
        T[:3, :3] = (U @ Vh).T
        T[:3, 3] = cb - T[:3, :3] @ ca
        if rmse < lowest:
            best, lowest = T.cpu(), rmse
    return best.numpy(), lowest


def exact(case, seed):
    kind = case["kind"]
    if kind == "preprocess":
        p = _points(case, _sequence(case, seed, 1)[1][0])
        return dict(pcd=p, normals=_normals(p))
    if kind == "icp":
        T, rmse = _icp(case, *_icp_pair(case, seed), case["plane"])
        return dict(T=T, rmse=np.float64(rmse))
    if kind == "dropin":
        poses, depth, _, g = _sequence(case, seed, 6, color=case["color"])
        start = [_small_motion(g, 0.5, 0.005) @ T for T in poses]
        T, rmse = _icp(case, depth[1], depth[0], start[1], poses[0], case["plane"])
        out = dict(pcd=None, T=T, rmse=np.float64(rmse))
        return dict(out, color=None) if case["color"] else out
    return None  # views, tracked poses, losses and meshes of a fused volume: see the module's comment
