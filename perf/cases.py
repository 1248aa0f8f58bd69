"""Measured cases of the distance-field collision engine: the calls a user's program makes, over the sizes it makes
them at.

    listed()                 the named cases
    draw(rng)                one more case of the same ranges
    prepare(case, seed)      what the program holds before the call: maps, clouds, queries, all made from the seed
    run(state)               one pass through the public entry points; its outputs
    work(case)               bytes and operations the pass cannot do without
    tolerance(case)          how far another correct implementation may be off
    exact(case, seed)        the same outputs from plain torch in 64 bits

A case's "kind" picks the path:

    frame      clear + insert + exact EDT of one sensor frame in one call, then squared-distance queries at voxel ids
    rebuild    the same frame as gpu-voxels programs write it: clearMap, insertPointCloud, parallelBanding3D, getDistances
    merge      a probabilistic map fed with a cloud, merged into a distance map, transformed
    batch      many maps of uneven dims in one schedule: clear + insert + EDT + trilinear distance and gradient queries
    maps       BitVectorVoxelMap against BitVectorVoxelMap: collision count and marks
    lists      many swept-volume lists against one environment map in one call: a count per list
    sweep      one swept volume: its voxel list built from a cloud, then collided with the environment map
    check      a robot's voxel list against the environment map: the count a control loop waits for
    trilinear  continuous distance + spatial gradient at points, and the adjoint for upstream gradients
    clearance  minimal clearance of a sphere-modelled arm per configuration
    traj       hinge cost of whole trajectories and its gradient, through autograd
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(_ROOT, "gpu-voxels_b200") not in sys.path:
    sys.path.insert(0, os.path.join(_ROOT, "gpu-voxels_b200"))

import gvx  # noqa: E402
from gvx import autograd  # noqa: E402
from gvx.batch import Batch  # noqa: E402

N_JOINTS, SPHERES_PER_LINK, MARGIN = 7, 8, 0.05


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: a control loop asks whether the robot's few thousand voxels meet the environment
        {"name": "check_64", "kind": "check", "x": 64, "y": 64, "z": 64, "scene": "boxes", "points": 6000, "n": 2000},
        # a workspace-sized field at 1 cm, rebuilt and queried at the configurations of one planning step
        {"name": "frame_128", "kind": "frame", "x": 128, "y": 128, "z": 128, "scene": "boxes", "points": 50_000,
         "n": 100_000},
        # the largest field: four 640 x 480 depth images into 512^3 at 5 mm
        {"name": "frame_512", "kind": "frame", "x": 512, "y": 512, "z": 512, "scene": "depth", "points": 1_228_800,
         "n": 100_000},
        # dims that are multiples of nothing (a room cut to its own extent), in the reference's three calls
        {"name": "rebuild_ragged", "kind": "rebuild", "x": 203, "y": 331, "z": 157, "scene": "boxes",
         "points": 150_000, "n": 20_000},
        # a mobile robot's flat map: sensor cloud -> probabilistic map -> distance field
        {"name": "merge_flat", "kind": "merge", "x": 320, "y": 320, "z": 96, "scene": "depth", "points": 307_200, "n": 0},
        # many workcells at once, dims log-uniform in [64, 384] per axis, 10k to 1M points each
        {"name": "batch_24", "kind": "batch", "maps": 24, "lo": 64, "hi": 384, "layout": 10, "n": 10_000},
        # whole-map collision of a depth scene with another map (capsule-like sparse bodies)
        {"name": "maps_384", "kind": "maps", "x": 384, "y": 384, "z": 384, "scene": "depth", "points": 900_000,
         "n": 200_000},
        # a planner's roadmap: thousands of swept-volume lists of 2k to 200k ids against one 256^3 environment
        {"name": "lists_1024", "kind": "lists", "x": 256, "y": 256, "z": 256, "scene": "boxes", "points": 50_000,
         "lists": 1024, "lo": 2000, "hi": 200_000, "mark": False},
        # one motion's swept volume voxelised into a list and checked
        {"name": "sweep_200k", "kind": "sweep", "x": 256, "y": 256, "z": 256, "scene": "boxes", "points": 50_000,
         "n": 200_000},
        # an optimiser's query batch: distance, gradient and adjoint at a million points
        {"name": "trilinear_1m", "kind": "trilinear", "x": 256, "y": 256, "z": 256, "scene": "boxes", "points": 50_000,
         "n": 1_000_000},
        # a sampling planner's batch of arm configurations, 56 spheres each
        {"name": "clearance_4096", "kind": "clearance", "x": 256, "y": 256, "z": 256, "scene": "boxes",
         "points": 50_000, "n": 4096},
        # a trajectory optimiser's step: 512 trajectories x 64 waypoints x 56 spheres, cost and gradient
        {"name": "traj_512", "kind": "traj", "x": 256, "y": 256, "z": 256, "scene": "boxes", "points": 50_000, "n": 512,
         "waypoints": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "rebuild", "merge", "batch", "maps", "lists", "sweep", "check", "trilinear",
                       "clearance", "traj"])
    c = {"kind": kind}
    if kind == "batch":
        return {"kind": kind, "maps": rng.randint(2, 24), "lo": 64, "hi": rng.randint(96, 320),
                "layout": rng.randint(0, 1 << 20), "n": _log_int(rng, 1000, 10_000)}
    top = {"frame": 448, "rebuild": 400, "merge": 320, "maps": 352, "lists": 256, "sweep": 320, "check": 192,
           "trilinear": 320, "clearance": 320, "traj": 320}[kind]
    low = 96 if kind in ("trilinear", "clearance", "traj") else 48
    for a in "xyz":
        c[a] = _log_int(rng, low, top)
    if rng.random() < 0.3:  # a program that rounds its dims up
        for a in "xyz":
            c[a] = (c[a] + 31) // 32 * 32
    c["scene"] = rng.choice(["boxes", "depth"]) if kind in ("frame", "rebuild", "merge", "maps") else "boxes"
    c["points"] = _log_int(rng, 5000, 600_000) if kind in ("frame", "rebuild", "merge", "maps") else 50_000
    if kind in ("frame", "rebuild"):
        c["n"] = _log_int(rng, 1000, 200_000)
    elif kind == "merge":
        c["n"] = 0
    elif kind == "maps":
        c["n"] = _log_int(rng, 5000, 200_000)
    elif kind == "lists":
        c["lists"] = _log_int(rng, 16, 1024)
        c["lo"] = 2000
        c["hi"] = _log_int(rng, 4000, 150_000)
        c["mark"] = rng.random() < 0.5
    elif kind == "sweep":
        c["n"] = _log_int(rng, 2000, 200_000)
    elif kind == "check":
        c["n"] = _log_int(rng, 500, 50_000)
    elif kind == "trilinear":
        c["n"] = _log_int(rng, 1000, 1_000_000)
    elif kind == "clearance":
        c["n"] = _log_int(rng, 16, 16_384)
    elif kind == "traj":
        c["n"] = _log_int(rng, 4, 512)
        c["waypoints"] = rng.choice([16, 33, 50, 64])
    return c


# ---------------------------------------------------------------------------
# inputs, made on the GPU from a seeded generator
# ---------------------------------------------------------------------------

def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _uniform(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _dims(case):
    return (case["x"], case["y"], case["z"])


def _side(case):
    return 0.005 if max(_dims(case)) > 320 else 0.01


def _boxes_cloud(g, extent, n, n_boxes=40, outliers=0.05):
    """Surface samples of random boxes (edges 4 % to 23 % of the extent) plus uniform outliers."""
    e = torch.as_tensor(extent, dtype=torch.float64, device="cuda")
    n_out = int(round(n * outliers))
    m = n - n_out
    edges = _uniform(g, n_boxes, 3, lo=0.05 / 1.28, hi=0.30 / 1.28) * e
    lo = _uniform(g, n_boxes, 3) * (e - edges)
    faces = torch.stack([edges[:, 1] * edges[:, 2], edges[:, 0] * edges[:, 2], edges[:, 0] * edges[:, 1]], 1)
    weight = torch.cat([faces, faces], 1).reshape(-1)  # box-major: axes 0..2 of the low faces, then of the high ones
    pick = torch.searchsorted(torch.cumsum(weight / weight.sum(), 0), _uniform(g, m)).clamp_(max=6 * n_boxes - 1)
    box, face = pick // 6, pick % 6
    p = lo[box] + _uniform(g, m, 3) * edges[box]
    axis = (face % 3)[:, None]
    flat = torch.where((face >= 3)[:, None], (lo + edges)[box], lo[box])
    p.scatter_(1, axis, flat.gather(1, axis))
    return torch.cat([p, _uniform(g, n_out, 3) * e]).float().contiguous()


def _depth_cloud(g, extent, n):
    """Floor and boxes seen by four pinhole cameras of 4:3 images (noise 2 mm per 2.56 m of extent)."""
    e = torch.as_tensor(extent, dtype=torch.float64, device="cuda")
    size = e[:2].mean()
    per = max(1, n // 4)
    width = max(4, int(round(math.sqrt(per * 4 / 3))))
    height = max(3, per // width)
    floor_z = 0.04 * e[2]
    edges = torch.stack([_uniform(g, 25, lo=0.02, hi=0.2) * e[0], _uniform(g, 25, lo=0.02, hi=0.2) * e[1],
                         _uniform(g, 25, lo=0.02, hi=0.2) * e[2]], 1)
    lo = torch.cat([_uniform(g, 25, 2) * (e[:2] - edges[:, :2]), floor_z.expand(25, 1)], 1)
    hi = lo + edges
    v, u = torch.meshgrid(torch.arange(height, device="cuda", dtype=torch.float64),
                          torch.arange(width, device="cuda", dtype=torch.float64), indexing="ij")
    f = 525.0 / 640.0 * width
    ray = torch.stack([(u - (width - 1) / 2) / f, (v - (height - 1) / 2) / f, torch.ones_like(u)], -1).reshape(-1, 3)
    target = torch.stack([e[0] / 2, e[1] / 2, floor_z])
    clouds = []
    for k in range(4):
        phi = 2 * math.pi * k / 4 + math.pi / 4
        eye = torch.stack([e[0] / 2 + 0.47 * e[0] * math.cos(phi), e[1] / 2 + 0.47 * e[1] * math.sin(phi), 0.6 * e[2]])
        z = (target - eye) / torch.linalg.norm(target - eye)
        x = torch.linalg.cross(z, torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda"))
        x = x / torch.linalg.norm(x)
        rot = torch.stack([x, torch.linalg.cross(z, x), z], 1)
        d = ray @ rot.T
        inv = 1.0 / torch.where(d.abs() < 1e-12, torch.full_like(d, 1e-12), d)
        t = torch.where(d[:, 2] < 0, (floor_z - eye[2]) * inv[:, 2], torch.full_like(d[:, 2], math.inf))
        for b in range(25):
            t0, t1 = (lo[b] - eye) * inv, (hi[b] - eye) * inv
            near, far = torch.minimum(t0, t1).amax(1), torch.maximum(t0, t1).amin(1)
            t = torch.where((far >= near) & (far > 0), torch.minimum(t, near.clamp(min=0)), t)
        ok = torch.isfinite(t)
        depth = t[ok] + torch.randn(int(ok.sum()), generator=g, device="cuda", dtype=torch.float64) * (0.002 / 2.56) * size
        clouds.append((ray[ok] * depth[:, None]) @ rot.T + eye)
    return torch.cat(clouds).float().contiguous()


def _cloud(case, seed, salt=1):
    extent = [d * _side(case) for d in _dims(case)]
    g = _gen(seed, salt)
    return _depth_cloud(g, extent, case["points"]) if case["scene"] == "depth" else _boxes_cloud(g, extent, case["points"])


def _bodies(case, seed, n, salt=2):
    """Points of a few compact bodies (a robot's links): 12 ellipsoids in a box of 0.7 times the map.  The bodies
    are the case's own; the seed moves the group by whole voxels and the points inside their voxels, so every seed
    occupies the same number of voxels."""
    rng = np.random.default_rng([n, *_dims(case)])
    box = np.maximum((0.7 * np.asarray(_dims(case))).astype(int), 1)
    centre, radii = rng.uniform(0.2, 0.8, (12, 3)) * box, rng.uniform(0.04, 0.15, (12, 3)) * box
    which, d = rng.integers(0, 12, n), rng.normal(size=(n, 3))
    d *= rng.uniform(size=(n, 1)) ** (1 / 3) / np.linalg.norm(d, axis=1, keepdims=True)
    voxel = np.clip(np.floor(centre[which] + d * radii[which]), 0, box - 1)
    g = _gen(seed, salt)
    move = (_uniform(g, 3) * torch.as_tensor(np.asarray(_dims(case)) - box + 1, device="cuda")).floor()
    p = torch.as_tensor(voxel, device="cuda") + move + _uniform(g, n, 3, lo=0.1, hi=0.9)
    return (p * _side(case)).float().contiguous()


def _batch_layout(case):
    """Dims and point counts of a batch's maps: the case's own, whatever the seed."""
    rng = np.random.default_rng(case["layout"])
    dims = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), size=(case["maps"], 3))).round().astype(int)
    pts = np.exp(rng.uniform(math.log(10_000), math.log(1_000_000), size=case["maps"])).round().astype(int)
    return [tuple(int(v) for v in d) for d in dims], [int(p) for p in pts]


def _list_lengths(case):
    rng = np.random.default_rng(case["lists"])
    return np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), size=case["lists"])).round().astype(np.int64)


def _csr_lists(case, seed):
    """Sorted unique ids per list (CSR).  A list's ids lie in a box of its own, as a swept volume's do."""
    g = _gen(seed, 3)
    X, Y, Z = _dims(case)
    length = torch.as_tensor(_list_lengths(case), device="cuda")
    k = length.shape[0]
    owner = torch.repeat_interleave(torch.arange(k, device="cuda"), length)
    full = torch.tensor([X, Y, Z], dtype=torch.float64, device="cuda")
    part = (length.double()[:, None] * 3 / full.prod()).clamp(max=1.0) ** (1 / 3)  # about 3 draws' room per id
    size = (part * full).ceil().clamp(min=2).minimum(full)
    low = (_uniform(g, k, 3) * (full - size + 1)).floor()
    ids = torch.zeros(owner.shape[0], dtype=torch.int64, device="cuda")
    for a, stride in ((0, 1), (1, X), (2, X * Y)):
        c = (low[owner, a] + (torch.rand(owner.shape[0], generator=g, device="cuda", dtype=torch.float64)
                              * size[owner, a]).floor()).long()
        ids += c * stride
    key = torch.unique(owner * (1 << 32) + ids)
    owner = key >> 32
    offsets = torch.zeros(k + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.cumsum(torch.bincount(owner, minlength=k), 0)
    return (key & 0xFFFFFFFF).to(torch.int32).contiguous(), offsets


def _arm(case):
    """A 7-joint arm with 8 spheres per link, scaled to the map."""
    rng = np.random.default_rng(4)
    extent = np.asarray(_dims(case)) * _side(case)
    scale = float(extent.min()) / 2.56
    a = rng.uniform(0.1, 0.4, size=N_JOINTS) * scale
    d = rng.uniform(0.1, 0.4, size=N_JOINTS) * scale
    alpha = rng.choice(np.array([math.pi / 2, -math.pi / 2, 0.0]), size=N_JOINTS)
    base = np.eye(4)
    base[:3, 3] = [extent[0] / 2, extent[1] / 2, 0.04 * extent[2]]
    n = N_JOINTS * SPHERES_PER_LINK
    return {"n_joints": N_JOINTS, "base": base.reshape(-1).tolist(), "theta": [0.0] * N_JOINTS, "d": d.tolist(),
            "a": a.tolist(), "alpha": alpha.tolist(), "link": [s // SPHERES_PER_LINK for s in range(n)],
            "t": [((s % SPHERES_PER_LINK) + 0.5) / SPHERES_PER_LINK for s in range(n)],
            "r": (rng.uniform(0.03, 0.08, size=n) * scale).tolist()}


def _configs(case, seed):
    g = _gen(seed, 5)
    if case["kind"] == "clearance":
        return _uniform(g, case["n"], N_JOINTS, lo=-math.pi, hi=math.pi).float().contiguous()
    q0, q1 = (_uniform(g, case["n"], 1, N_JOINTS, lo=-math.pi, hi=math.pi) for _ in range(2))
    t = torch.linspace(0, 1, case["waypoints"], device="cuda", dtype=torch.float64)[None, :, None]
    return (q0 + (q1 - q0) * t).float().contiguous()


def _query_points(case, seed):
    g = _gen(seed, 6)
    d = torch.as_tensor(_dims(case), dtype=torch.float64, device="cuda")
    side = _side(case)
    return (0.5 * side + _uniform(g, case["n"], 3) * (d - 1) * side).float().contiguous()


def _ids(case, seed):
    n = case["x"] * case["y"] * case["z"]
    return torch.randint(0, n, (case["n"],), generator=_gen(seed, 7), device="cuda").to(torch.int32)


def _held(owner, view):
    """A map's borrowed view of its device memory, holding the map: the outputs of a pass outlive the state."""
    view.owner = owner
    return view


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": dict(case)}
    if kind == "batch":
        dims, counts = _batch_layout(case)
        side = 0.01
        clouds = [_boxes_cloud(_gen(seed, 20 + k), [v * side for v in d], n) for k, (d, n) in enumerate(zip(dims, counts))]
        s["maps"] = [gvx.DistanceVoxelMap(d, side) for d in dims]
        s["fields"] = [_held(m, m.data()) for m in s["maps"]]
        s["xyz"] = torch.cat(clouds)
        s["offsets"] = torch.tensor([0] + np.cumsum([c.shape[0] for c in clouds]).tolist(), device="cuda")
        g = _gen(seed, 9)
        s["q"] = torch.cat([(0.5 * side + _uniform(g, case["n"], 3) * (torch.tensor(d, device="cuda").double() - 1) * side)
                            for d in dims]).float().contiguous()
        s["q_map"] = torch.arange(len(dims), device="cuda", dtype=torch.int32).repeat_interleave(case["n"])
        s["batch"] = Batch(s["maps"])
        return s
    dims, side = _dims(case), _side(case)
    if kind in ("frame", "rebuild", "merge"):
        s["cloud"] = _cloud(case, seed)
        s["map"] = gvx.DistanceVoxelMap(dims, side)
        s["field"] = _held(s["map"], s["map"].data())
        if kind == "merge":
            s["prob"] = gvx.ProbVoxelMap(dims, side)
            s["occ"] = _held(s["prob"], s["prob"].data())
        else:
            s["ids"] = _ids(case, seed)
        return s
    if kind in ("maps", "lists", "sweep", "check"):
        s["env"] = gvx.BitVectorVoxelMap(dims, side)
        s["env"].insertPointCloud(_cloud(case, seed), gvx.eBVM_OCCUPIED)
    if kind == "maps":
        s["body"] = gvx.BitVectorVoxelMap(dims, side)
        s["body"].insertPointCloud(_bodies(case, seed, case["n"]), 4)
        s["marks"] = _held(s["body"], s["body"].voxels())
    elif kind == "lists":
        s["ids"], s["offsets"] = _csr_lists(case, seed)
        s["voxels"] = torch.zeros(s["ids"].shape[0], 32, dtype=torch.uint8, device="cuda")
        s["voxels"][:, 0] = 16  # swept-volume meaning 4
    elif kind == "sweep":
        s["list"] = gvx.BitVectorVoxelList(dims, side)
        s["cloud"] = _bodies(case, seed, case["n"])
    elif kind == "check":
        s["list"] = gvx.BitVectorVoxelList(dims, side)
        s["list"].insertPointCloud(_bodies(case, seed, case["n"]), 4)
    elif kind in ("trilinear", "clearance", "traj"):
        s["map"] = gvx.DistanceVoxelMap(dims, side)
        s["map"].voxelize_edt(_cloud(case, seed))
        if kind == "trilinear":
            s["q"] = _query_points(case, seed)
            s["up"] = torch.randn(case["n"], generator=_gen(seed, 8), device="cuda")
        else:
            s["arm"] = gvx.make_arm(_arm(case))
            s["q"] = _configs(case, seed)
            if kind == "traj":
                autograd.build()
                s["q"].requires_grad_(True)
                s["up"] = torch.rand(case["n"], generator=_gen(seed, 8), device="cuda") + 0.5
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "frame":
        s["map"].voxelize_edt(s["cloud"])
        return s["field"], s["map"].getSquaredDistances(s["ids"])
    if kind == "rebuild":
        s["map"].clearMap()
        s["map"].insertPointCloud(s["cloud"])
        s["map"].parallelBanding3D()
        return s["field"], s["map"].getDistances(s["ids"])
    if kind == "merge":
        s["prob"].clearMap()
        s["prob"].insertPointCloud(s["cloud"])
        s["map"].clearMap()
        s["map"].mergeOccupied(s["prob"], (0, 0, 0), 0.6)
        s["map"].parallelBanding3D()
        return s["occ"], s["field"]
    if kind == "batch":
        s["batch"].voxelize_edt(s["xyz"], s["offsets"])
        dist, grad = s["batch"].query(s["q"], s["q_map"])
        return s["fields"], dist, grad
    if kind == "maps":
        return s["body"].collideWith(s["env"]), s["marks"]
    if kind == "lists":
        counts = gvx.lists_collide_map(s["ids"], s["voxels"], s["offsets"], s["env"], mark=s["case"]["mark"])
        return (counts, s["voxels"]) if s["case"]["mark"] else counts
    if kind == "sweep":
        s["list"].clearMap()
        s["list"].insertPointCloud(s["cloud"], 4)
        return s["list"].collideWith(s["env"]), s["list"].ids(), s["list"].voxels()
    if kind == "check":
        return s["list"].collideWith(s["env"]), s["list"].voxels()
    if kind == "trilinear":
        dist, grad = s["map"].trilinear(s["q"])
        return dist, grad, s["map"].trilinear_backward(s["q"], s["up"])
    if kind == "clearance":
        return s["map"].sphere_clearance(s["arm"], s["q"])
    cost = autograd.trajectory_cost(s["q"], s["map"], s["arm"], MARGIN)
    (grad,) = torch.autograd.grad(cost, s["q"], s["up"])
    return cost.detach(), grad


def work(case):
    kind = case["kind"]
    if kind == "batch":
        dims, counts = _batch_layout(case)
        vox = sum(x * y * z for x, y, z in dims)
        n = case["n"] * len(dims)
        return {"bytes": 4 * vox + 12 * sum(counts) + n * (12 + 4 + 32 + 16), "flops": 60 * n}
    vox = case["x"] * case["y"] * case["z"]
    n = case.get("n", 0)
    if kind in ("frame", "rebuild"):  # points in, the field out; id, voxel and answer per query
        return {"bytes": 4 * vox + 12 * case["points"] + 12 * n, "flops": 6 * n}
    if kind == "merge":
        return {"bytes": 5 * vox + 12 * case["points"], "flops": 0}
    if kind == "maps":
        return {"bytes": 64 * vox, "flops": 0}
    if kind == "lists":
        ids = int(_list_lengths(case).sum())
        return {"bytes": 32 * vox + 4 * ids + 8 * case["lists"], "flops": 0}
    if kind == "sweep":  # the points, the list written, each entry's voxel of the map; duplicates merge
        return {"bytes": 12 * n + 36 * n + 32 * n, "flops": 0}
    if kind == "check":
        return {"bytes": (4 + 32 + 32) * n, "flops": 0}
    if kind == "trilinear":  # forward: point, 8 corners, distance, gradient; adjoint: point, corners, upstream, gradient
        return {"bytes": n * (12 + 32 + 16 + 12 + 32 + 4 + 12), "flops": 120 * n}
    spheres = N_JOINTS * SPHERES_PER_LINK
    if kind == "clearance":
        return {"bytes": n * (4 * N_JOINTS + 4 + spheres * 32), "flops": n * (spheres * 70 + N_JOINTS * 120)}
    wp = n * case["waypoints"]
    return {"bytes": wp * (2 * 4 * N_JOINTS + 4 * N_JOINTS + 2 * spheres * 32) + 8 * n,
            "flops": wp * (2 * spheres * 70 + 2 * N_JOINTS * 120 + spheres * 4 * 18)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("batch", "trilinear"):  # FP32 interpolation of exact corner distances (7e-7 off 64 bits)
        return {"rel": 2.5e-6, "max": 5e-5}
    if kind == "clearance":  # one interpolated distance per output (3e-8 off)
        return {"rel": 3e-7, "max": 3e-6}
    if kind == "traj":
        # The gradient jumps where a sphere's centre crosses a cell face: another rounding of the kinematics puts one
        # of 1.8 million centres into the next cell (9e-4 off 64 bits where that happens, 3e-7 where it does not).
        return {"rel": 3.5e-3}
    return "exact"


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain torch
# ---------------------------------------------------------------------------

def _voxel_of(p, side):
    """Voxel coordinates as single precision defines them (the input's own type)."""
    return torch.floor(p / torch.tensor(side, dtype=torch.float32, device=p.device)).long()


def _occupied(dims, side, cloud):
    v = _voxel_of(cloud, side).clamp_(min=0)  # negative coordinates land in voxel 0
    ok = (v < torch.tensor(dims, device="cuda")).all(1)
    v = v[ok]
    occ = torch.zeros(dims[2], dims[1], dims[0], dtype=torch.bool, device="cuda")
    occ[v[:, 2], v[:, 1], v[:, 0]] = True
    return occ


def _squared_distances(occ):
    """Exact squared distance to the nearest occupied voxel, axis by axis (int32 holds it)."""
    far = 1 << 29
    d = torch.where(occ, 0, far).to(torch.int32)
    for axis in range(3):
        n = d.shape[axis]
        r = torch.arange(n, device="cuda", dtype=torch.int32)
        out = d.clone()
        shape = [1, 1, 1]
        shape[axis] = n
        for j in range(n):
            out = torch.minimum(out, d.narrow(axis, j, 1) + ((r - j) ** 2).reshape(shape))
        d = out
    return torch.where(d >= far, torch.full_like(d, 2147483647), d)


def _trilinear64(sq, side, p):
    """Distance (metres) and gradient of the trilinear interpolant at points p (float64), sq[z, y, x]."""
    Z, Y, X = sq.shape
    n = torch.tensor([X, Y, Z], dtype=torch.float64, device="cuda")
    u = p / side - 0.5
    free = (u >= 0) & (u <= n - 1)
    uc = torch.minimum(u.clamp(min=0), n - 1)
    i0 = torch.minimum(uc.floor(), (n - 2).clamp(min=0)).long()
    f = uc - i0
    i1 = torch.minimum(i0 + 1, (n - 1).long())
    x, y, z = ((i0[:, a], i1[:, a]) for a in range(3))
    c = [[[sq[z[k], y[j], x[i]].double().sqrt() for i in (0, 1)] for j in (0, 1)] for k in (0, 1)]
    fx, fy, fz = f[:, 0], f[:, 1], f[:, 2]
    mix = lambda a, b, t: a + (b - a) * t  # noqa: E731
    e = [[mix(c[k][j][0], c[k][j][1], fx) for j in (0, 1)] for k in (0, 1)]
    s = [mix(e[k][0], e[k][1], fy) for k in (0, 1)]
    dx = mix(mix(c[0][0][1] - c[0][0][0], c[0][1][1] - c[0][1][0], fy),
             mix(c[1][0][1] - c[1][0][0], c[1][1][1] - c[1][1][0], fy), fz)
    dy = mix(e[0][1] - e[0][0], e[1][1] - e[1][0], fz)
    grad = torch.stack([dx, dy, s[1] - s[0]], 1) * free
    return mix(s[0], s[1], fz) * side, grad


def _chain64(arm, q):
    """Joint frames of the DH chain, FP64: origins [N, J + 1, 3] and joint axes [N, J, 3].  Every arm parameter is
    the float32 value that the call gets."""
    f32 = lambda v: torch.tensor(v, dtype=torch.float32, device="cuda").double()  # noqa: E731
    base = f32(arm["base"]).reshape(4, 4)
    r = base[:3, :3].expand(q.shape[0], 3, 3)
    o = base[:3, 3].expand(q.shape[0], 3)
    d, a, alpha, theta = (f32(arm[k]) for k in ("d", "a", "alpha", "theta"))
    origins, axes = [o], []
    for j in range(arm["n_joints"]):
        axes.append(r[:, :, 2])
        th = q[:, j].double() + theta[j]
        ct, st = th.cos(), th.sin()
        ca, sa = alpha[j].cos(), alpha[j].sin()
        zero = torch.zeros_like(ct)
        step = torch.stack([ct, -st * ca, st * sa, st, ct * ca, -ct * sa, zero, sa.expand_as(ct), ca.expand_as(ct)],
                           1).reshape(-1, 3, 3)
        shift = torch.stack([a[j] * ct, a[j] * st, d[j].expand_as(ct)], 1)
        o = (r @ shift[:, :, None])[:, :, 0] + o
        r = r @ step
        origins.append(o)
    return torch.stack(origins, 1), torch.stack(axes, 1)


def _spheres64(arm, origins):
    link = torch.tensor(arm["link"], device="cuda")
    t = torch.tensor(arm["t"], dtype=torch.float32, device="cuda").double()[None, :, None]
    lo, hi = origins[:, link], origins[:, link + 1]
    return lo + (hi - lo) * t, torch.tensor(arm["r"], dtype=torch.float32, device="cuda").double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        dims, counts = _batch_layout(case)
        if sum(x * y * z * (x + y + z) for x, y, z in dims) > 2.5e11:
            return None
        side = 0.01
        f32 = float(np.float32(side))
        g = _gen(seed, 9)
        dist, grad = [], []
        for k, (d, n) in enumerate(zip(dims, counts)):
            sq = _squared_distances(_occupied(d, side, _boxes_cloud(_gen(seed, 20 + k), [v * side for v in d], n)))
            q = (0.5 * side + _uniform(g, case["n"], 3) * (torch.tensor(d, device="cuda").double() - 1) * side).float()
            a, b = _trilinear64(sq, f32, q.double())
            dist.append(a)
            grad.append(b)
        return [None] * len(dims), torch.cat(dist), torch.cat(grad)
    dims, side = _dims(case), _side(case)
    f32 = float(np.float32(side))
    if kind in ("frame", "rebuild"):
        sq = _squared_distances(_occupied(dims, side, _cloud(case, seed))).reshape(-1)[_ids(case, seed).long()]
        return None, sq if kind == "frame" else sq.double().sqrt().floor().to(torch.int32)
    if kind == "merge":
        return None
    if kind in ("maps", "sweep", "check"):
        env = _occupied(dims, side, _cloud(case, seed)).reshape(-1)
        body = _occupied(dims, side, _bodies(case, seed, case["n"])).reshape(-1)
        ids = body.nonzero()[:, 0]
        count = int((env & body).sum())
        if kind == "maps":
            return count, None
        return (count, ids.to(torch.int32), None) if kind == "sweep" else (count, None)
    if kind == "lists":
        env = _occupied(dims, side, _cloud(case, seed)).reshape(-1)
        ids, offsets = _csr_lists(case, seed)
        run_sum = torch.zeros(ids.shape[0] + 1, dtype=torch.int64, device="cuda")
        run_sum[1:] = torch.cumsum(env[ids.long()].long(), 0)
        counts = run_sum[offsets[1:]] - run_sum[offsets[:-1]]
        return (counts, None) if case["mark"] else counts
    sq = _squared_distances(_occupied(dims, side, _cloud(case, seed)))
    if kind == "trilinear":
        dist, grad = _trilinear64(sq, f32, _query_points(case, seed).double())
        up = torch.randn(case["n"], generator=_gen(seed, 8), device="cuda").double()
        return dist, grad, grad * up[:, None]
    arm, q = _arm(case), _configs(case, seed)
    if kind == "clearance":
        origins, _ = _chain64(arm, q)
        c, r = _spheres64(arm, origins)
        d, _ = _trilinear64(sq, f32, c.reshape(-1, 3))
        return (d.reshape(c.shape[:2]) - r).amin(1)
    margin = float(np.float32(MARGIN))
    cost, grads = [], []
    link = torch.tensor(arm["link"], device="cuda")
    moves = (torch.arange(N_JOINTS, device="cuda")[None, :] <= link[:, None]).double()  # joints that move a sphere
    for part in q.split(64):  # the chain rule by hand, a few trajectories at a time
        flat = part.reshape(-1, N_JOINTS)
        origins, axes = _chain64(arm, flat)
        c, r = _spheres64(arm, origins)
        d, g = _trilinear64(sq, f32, c.reshape(-1, 3))
        hinge = margin - (d.reshape(c.shape[:2]) - r)
        cost.append(hinge.clamp(min=0).reshape(part.shape[0], -1).sum(1))
        g = g.reshape(c.shape) * (hinge > 0)[:, :, None]
        arm_to = c[:, :, None, :] - origins[:, None, :-1, :]
        turn = torch.linalg.cross(axes[:, None].expand_as(arm_to), arm_to)
        grads.append((-(turn * g[:, :, None, :]).sum(-1) * moves).sum(1).reshape(part.shape))
    up = (torch.rand(case["n"], generator=_gen(seed, 8), device="cuda") + 0.5).double()
    return torch.cat(cost), torch.cat(grads) * up[:, None, None]
