"""Timed cases of this framework: what its users run, over the range of sizes they run it on.

* ``forward``: ``PointTransformerV3`` on a batch of voxelised scenes, from one small room (an
  interactive tool, where launches and host work count) to a batch of LiDAR sweeps (a scoring job);
* ``segment``: raw points -> ``voxelize`` -> backbone -> ``SegHead`` -> logits of every raw point;
* ``serialize``: ``Point.serialization`` in all four orders, for code that sorts clouds and brings
  its own network;
* ``attention``, ``xcpe``: one ``SerializedAttention`` / one 3x3x3 ``SubMConv3d`` with its kernel map,
  for code that builds its own blocks;
* ``voxelize``: the front end alone, as a data loader runs it.

Scenes are synthetic, made on the GPU from the seed: rectangles in a room (walls, floors, table tops)
and a spinning multi-beam LiDAR over a ground plane with boxes.  Sizes follow the benchmark's
configurations; scenes of one batch differ in size, as scans do.
"""
import math

import torch

from pointtransformerv3_b200 import Point, PointTransformerV3, SegHead, SerializedAttention, SubMConv3d, voxelize

ORDERS = ("z", "z-trans", "hilbert", "hilbert-trans")
CLASSES = 20                                    # labels of an indoor benchmark
ENC_DEPTHS, ENC_CHANNELS = (2, 2, 2, 6, 2), (32, 64, 128, 256, 512)
DEC_DEPTHS, DEC_CHANNELS = (2, 2, 2, 2), (64, 64, 128, 256)
# points of a level / points of the level above it, and occupied 3x3x3 neighbours (itself included), for `work`
POOLED = {"indoor": 0.26, "lidar": 0.45}
NEIGHBOURS = {"indoor": 8.8, "lidar": 5.0}
LIDAR_VOXELS = 64000                            # voxels of one 64-beam sweep at grid 0.05
RAW_PER_VOXEL = 6                               # raw points per occupied voxel of a room scan


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # one small room or object scan: launches, host work and read-backs are what its user waits for
        dict(name="forward_room_6k", path="forward", kind="indoor", scenes=1, size=6000, dtype="bf16", flash=True,
             stream=False),
        # one room scan, called and waited for: the ordinary interactive use
        dict(name="forward_room_100k", path="forward", kind="indoor", scenes=1, size=100000, dtype="bf16",
             flash=True, stream=False),
        # the benchmark's batch, fed by a loader that knows the batch on the host and reads the status word late
        dict(name="forward_4_rooms_100k", path="forward", kind="indoor", scenes=4, size=100000, dtype="bf16",
             flash=True, stream=True),
        # one LiDAR frame of two merged sweeps, as a robot runs it
        dict(name="forward_lidar_frame", path="forward", kind="lidar", scenes=1, size=2, dtype="bf16", flash=True,
             stream=False),
        # sixteen LiDAR frames at once: an offline scoring job, the largest batch of the benchmark
        dict(name="forward_16_lidar_frames", path="forward", kind="lidar", scenes=16, size=2, dtype="bf16",
             flash=True, stream=True),
        # 32-bit features with the patch rule of the non-flash path: reference results, ragged batch of two
        dict(name="forward_2_rooms_20k_fp32", path="forward", kind="indoor", scenes=2, size=20000, dtype="fp32",
             flash=False, stream=False),
        # from the sensor's points to logits per raw point, two rooms
        dict(name="segment_2_rooms", path="segment", kind="indoor", scenes=2, size=60000, dtype="bf16", flash=True,
             stream=False),
        # serialization alone: 100 000 uniform points, and a large aggregated cloud
        dict(name="serialize_100k", path="serialize", points=100000, extent=10.0, grid=0.02),
        dict(name="serialize_8m", path="serialize", points=8000000, extent=60.0, grid=0.02),
        # one attention module at the width of the finest decoder level
        dict(name="attention_120k", path="attention", points=120000, channels=64, patch=1024, dtype="bf16"),
        # kernel map + convolution of one positional encoding, 128 channels
        dict(name="xcpe_85k_128", path="xcpe", size=85000, channels=128, dtype="bf16"),
        # raw points of four room scans to one point per voxel
        dict(name="voxelize_2400k", path="voxelize", scenes=4, size=100000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(("forward",) * 6 + ("segment", "segment", "serialize", "attention", "xcpe", "voxelize"))
    if path == "forward":
        if rng.random() < 0.15:
            return dict(path=path, kind="indoor", scenes=rng.randint(1, 3), size=_log(rng, 2000, 30000), dtype="fp32",
                        flash=rng.random() < 0.3, stream=False)
        stream = rng.random() < 0.5
        flash = rng.random() < 0.85
        if rng.random() < 0.35:
            return dict(path=path, kind="lidar", scenes=_log(rng, 1, 15), size=rng.randint(1, 2), dtype="bf16",
                        flash=flash, stream=stream)
        total = _log(rng, 4000, 1200000)
        scenes = rng.randint(max(1, -(-total // 150000)), max(1, min(12, total // 3000)))
        return dict(path=path, kind="indoor", scenes=scenes, size=total // scenes, dtype="bf16", flash=flash,
                    stream=stream)
    if path == "segment":
        return dict(path=path, kind="indoor", scenes=rng.randint(1, 4), size=_log(rng, 4000, 120000), dtype="bf16",
                    flash=True, stream=False)
    if path == "serialize":
        n = _log(rng, 3001, 8000000)
        return dict(path=path, points=n, extent=round(rng.uniform(4.0, 80.0), 1), grid=rng.choice((0.02, 0.05)))
    if path == "attention":
        return dict(path=path, points=_log(rng, 3001, 400000), channels=rng.choice((32, 64, 128, 256)),
                    patch=rng.choice((256, 1024, 1024)), dtype="bf16")
    if path == "xcpe":
        return dict(path=path, size=_log(rng, 3001, 300000), channels=rng.choice((32, 64, 128, 256)), dtype="bf16")
    return dict(path=path, scenes=rng.randint(1, 4), size=_log(rng, 4000, 120000))


# --------------------------------------------------------------------------- scenes
# A case's sizes are exact whatever the seed: a scene is made somewhat too large and cut.
def _generators(seed):
    return torch.Generator().manual_seed(seed), torch.Generator(device="cuda").manual_seed(seed)


def _scene_sizes(case, size):
    """Points or voxels of every scene of a batch: 0.7 to 1.3 times the nominal size."""
    if case["scenes"] == 1:
        return [size]
    return [int(size * (0.7 + 0.6 * (0.618 * (i + 1) % 1.0))) | 1 for i in range(case["scenes"])]


def _cells(coord, grid_size):
    """(grid_coord (N, 3) int32, cell of every point, first point of every cell in input order)."""
    gc = torch.div(coord, torch.full_like(coord, grid_size), rounding_mode="trunc").int()     # a true division
    key = (gc[:, 0].long() << 42) | (gc[:, 1].long() << 21) | gc[:, 2].long()
    n = coord.shape[0]
    uniq, inv = torch.unique(key, return_inverse=True)
    first = torch.full((uniq.shape[0],), n, dtype=torch.int64, device=coord.device)
    first.scatter_reduce_(0, inv, torch.arange(n, device=coord.device), "amin")
    return gc, inv, first


def _room(host, dev, voxels, grid_size=0.02, n_rect=20):
    """(points, cells, first point of every cell) of a 10 x 10 x 3 m room with exactly ``voxels`` occupied
    cells: points on axis-aligned rectangles, rectangle after rectangle, the last ones cut off.  The first
    point is the room's corner, the origin of its grid."""
    room, spare = torch.tensor((10.0, 10.0, 3.0)), 1.3
    while True:
        s = math.sqrt(spare * voxels * grid_size ** 2 / (n_rect * 2.25))
        lo, side, axes, counts = torch.zeros(n_rect, 3), torch.zeros(n_rect, 3), [], []
        for i in range(n_rect):
            axis = i % 3
            a, b = [d for d in range(3) if d != axis]
            sd = torch.minimum((1.0 + torch.rand(2, generator=host)) * s, room[[a, b]])
            side[i, [a, b]] = sd
            lo[i, [a, b]] = torch.rand(2, generator=host) * (room[[a, b]] - sd)
            lo[i, axis] = torch.rand(1, generator=host) * room[axis]
            axes.append(a)
            counts.append(int((RAW_PER_VOXEL + 1) * sd[0] * sd[1] / grid_size ** 2))
        counts, axes = torch.tensor(counts, device="cuda"), torch.tensor(axes, device="cuda")
        rect = torch.arange(n_rect, device="cuda").repeat_interleave(counts)
        uv = torch.rand(rect.shape[0], 3, device="cuda", generator=dev)
        # along its first side a rectangle is scanned from one end to the other
        sweep = (torch.arange(rect.shape[0], device="cuda") - (counts.cumsum(0) - counts)[rect] + 0.5) / counts[rect]
        uv.scatter_(1, axes[rect][:, None], sweep[:, None].float())
        coord = torch.cat([torch.zeros(1, 3, device="cuda"), lo.cuda()[rect] + uv * side.cuda()[rect]])
        gc, inv, first = _cells(coord, grid_size)
        if first.shape[0] >= voxels:
            break
        spare *= 1.3
    keep = first.sort().values[:voxels]                        # cells in the order they were met
    kept = torch.zeros(first.shape[0], dtype=torch.bool, device="cuda")
    kept[inv[keep]] = True
    return coord, gc, keep, kept[inv]


def _room_voxels(host, dev, voxels):
    """(coord, grid_coord) of one point per cell, in random order."""
    coord, gc, keep, _ = _room(host, dev, voxels)
    keep = keep[torch.randperm(voxels, device="cuda", generator=dev)]
    return coord[keep], gc[keep]


def _room_points(host, dev, voxels):
    """RAW_PER_VOXEL x voxels points of a room in random order, every cell hit."""
    coord, _, keep, kept = _room(host, dev, voxels)
    kept[keep] = False
    others = kept.nonzero().squeeze(1)
    others = others[torch.randperm(others.shape[0], device="cuda", generator=dev)]
    pick = torch.cat([keep, others])[:RAW_PER_VOXEL * voxels]
    pick = torch.cat([pick, pick[:RAW_PER_VOXEL * voxels - pick.shape[0]]])
    return coord[pick[torch.randperm(pick.shape[0], device="cuda", generator=dev)]]


def _lidar_voxels(host, dev, voxels, sweeps, beams=64, steps=2048, max_range=50.0):
    """(coord, grid_coord) of one point per cell of merged sweeps of a spinning LiDAR (elevations -25..+3
    degrees) over a ground plane with 10-30 boxes, in scan order; the farthest rings are cut off."""
    n_box = 10 + int(torch.randint(0, 21, (1,), generator=host))
    centre = (torch.rand(n_box, 2, generator=host) - 0.5) * 80.0
    half = 0.5 + torch.rand(n_box, 3, generator=host) * torch.tensor([3.0, 3.0, 2.5])
    lo = torch.cat([centre - half[:, :2], torch.zeros(n_box, 1)], 1).cuda()
    hi = torch.cat([centre + half[:, :2], 2 * half[:, 2:]], 1).cuda()
    elev = torch.deg2rad(torch.linspace(-25.0, 3.0, beams, device="cuda"))[:, None].expand(-1, steps)
    azim = (torch.arange(steps, device="cuda") * (2 * math.pi / steps))[None, :].expand(beams, -1)
    d = torch.stack([elev.cos() * azim.cos(), elev.cos() * azim.sin(), elev.sin()], -1).reshape(-1, 3)
    inv_d = 1.0 / torch.where(d.abs() < 1e-9, torch.full_like(d, 1e-9), d)
    ray = torch.arange(d.shape[0], device="cuda")
    points, rays, s = [], [], 0
    while True:
        origin = torch.tensor([1.0 * s, 0.3 * s, 1.8], device="cuda")
        t = torch.where(d[:, 2] < -1e-6, -origin[2] / d[:, 2], torch.full_like(d[:, 2], math.inf))
        t0, t1 = (lo - origin)[:, None] * inv_d, (hi - origin)[:, None] * inv_d          # (boxes, rays, 3)
        near, far = torch.minimum(t0, t1).amax(2), torch.maximum(t0, t1).amin(2)
        hit = (near <= far) & (near > 0)
        t = torch.minimum(t, torch.where(hit, near, torch.full_like(near, math.inf)).amin(0))
        noise = 1.0 + 0.002 * torch.randn(d.shape[0], device="cuda", generator=dev)
        ok = t < max_range
        points.append((origin + d * (t * noise)[:, None])[ok])
        rays.append(ray[ok])
        s += 1
        if s < sweeps:
            continue
        coord = torch.cat(points)
        gc, _, first = _cells(coord - coord.min(0)[0], 0.05)
        if first.shape[0] >= voxels:
            break
    first = first.sort().values
    near_first = torch.cat(rays)[first].argsort(stable=True)[:voxels]       # rings from the sensor outwards
    keep = first[near_first.sort().values]
    gc = gc[keep]
    return coord[keep], gc - gc.amin(0)


def _batch(case, seed):
    """data_dict of a voxelised batch, with the host's copy of what a loader knows where it streams."""
    host, dev = _generators(seed)
    if case["kind"] == "indoor":
        scenes = [_room_voxels(host, dev, n) for n in _scene_sizes(case, case["size"])]
    else:
        scenes = [_lidar_voxels(host, dev, n, case["size"])
                  for n in _scene_sizes(case, case["size"] * LIDAR_VOXELS)]
    coord, grid = torch.cat([s[0] for s in scenes]), torch.cat([s[1] for s in scenes])
    # colour, or intensity
    extra = torch.rand(coord.shape[0], 3 if case["kind"] == "indoor" else 1, device="cuda", generator=dev)
    offset = torch.tensor([s[0].shape[0] for s in scenes]).cumsum(0)
    data = dict(coord=coord, grid_coord=grid, feat=torch.cat([coord, extra], 1).to(_dtype(case)),
                offset=offset.cuda())
    if case["stream"]:
        top = grid.amax(0).tolist()
        data.update(offset_host=offset.tolist(), sparse_shape=[v + 96 for v in top],
                    serialization_depth=max(top).bit_length())
    return data


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float32


def _network(case):
    """The default backbone with random weights (the same for every seed: a program keeps its weights)."""
    torch.manual_seed(7)
    with torch.device("cuda"):
        net = PointTransformerV3(in_channels=6 if case["kind"] == "indoor" else 4, enable_flash=case["flash"])
        head = SegHead(DEC_CHANNELS[0], CLASSES)
    net, head = net.to(_dtype(case)).eval(), head.to(_dtype(case)).eval()
    net.defer_status_check = case["stream"]
    return net, head


# --------------------------------------------------------------------------- prepare and run
@torch.no_grad()
def prepare(case, seed):
    path = case["path"]
    host, dev = _generators(seed)
    state = dict(case=case, path=path, seed=seed)
    if path == "forward":
        state["data"] = _batch(case, seed)
        state["net"], _ = _network(case)
    elif path == "segment" or path == "voxelize":
        clouds = [_room_points(host, dev, n) for n in _scene_sizes(case, case["size"])]
        state["coord"] = torch.cat(clouds)
        state["feat"] = torch.cat([state["coord"], torch.rand(state["coord"].shape[0], 3, device="cuda", generator=dev)],
                                  1)
        state["offset"] = torch.tensor([c.shape[0] for c in clouds]).cumsum(0).cuda()
        if path == "segment":
            state["feat"] = state["feat"].to(_dtype(case))
            state["net"], state["head"] = _network(case)
    elif path == "serialize":
        n = case["points"]
        xyz = torch.rand(n, 3, device="cuda", generator=dev) * case["extent"]
        state["grid"] = torch.div(xyz - xyz.min(0)[0], case["grid"], rounding_mode="trunc").int()
        state["offset"] = torch.tensor([n], device="cuda")
    elif path == "attention":
        n, c = case["points"], case["channels"]
        torch.manual_seed(7)
        with torch.device("cuda"):
            attn = SerializedAttention(c, c // 16, case["patch"], upcast_attention=False, upcast_softmax=False,
                                       order_index=0)
        state["attn"] = attn.to(_dtype(case)).eval()
        grid = torch.randint(0, 500, (n, 3), device="cuda", generator=dev, dtype=torch.int32)
        point = Point(feat=torch.randn(n, c, device="cuda", generator=dev).to(_dtype(case)), grid_coord=grid,
                      offset=torch.tensor([n], device="cuda"))
        point.serialization(order="hilbert")
        state["attn"].get_padding_and_inverse(point)          # a level's blocks share one patch layout
        state["point"] = point
    elif path == "xcpe":
        c = case["channels"]
        torch.manual_seed(7)
        with torch.device("cuda"):
            conv = SubMConv3d(c, c, kernel_size=3, bias=True, indice_key="cpe")
        state["conv"] = conv.to(_dtype(case)).eval()
        grid = _room_voxels(host, dev, case["size"])[1]
        point = Point(feat=torch.randn(grid.shape[0], c, device="cuda", generator=dev).to(_dtype(case)),
                      grid_coord=grid, offset=torch.tensor([grid.shape[0]], device="cuda"))
        point.serialization(order="z")
        state["point"] = point
    return state


@torch.inference_mode()
def run(state):
    path = state["path"]
    if path == "forward" or path == "segment":
        # the order shuffle of every pass comes from torch's CPU generator: seeded, as for a repeatable result
        torch.random.default_generator.manual_seed(state["seed"])
    if path == "forward":
        point = state["net"](dict(state["data"]))
        return {"feat": point.feat, "status": point["_status"]} if state["case"]["stream"] else point.feat
    if path == "segment":
        data, point2voxel = voxelize(state["coord"], state["feat"], state["offset"], 0.02)
        point = state["head"](state["net"](data))
        return {"logits": point.seg_logits[point2voxel], "point2voxel": point2voxel}
    if path == "voxelize":
        data, point2voxel = voxelize(state["coord"], state["feat"], state["offset"], 0.02)
        return {"coord": data["coord"], "grid_coord": data["grid_coord"], "feat": data["feat"],
                "offset": data["offset"], "point2voxel": point2voxel}
    if path == "serialize":
        point = Point(grid_coord=state["grid"], offset=state["offset"])
        point.serialization(order=ORDERS)
        return {"code": point.serialized_code, "order": point.serialized_order, "inverse": point.serialized_inverse}
    if path == "attention":
        return state["attn"](Point(state["point"])).feat
    point = Point(state["point"])
    point.sparsify()
    return state["conv"](point.sparse_conv_feat).features


# --------------------------------------------------------------------------- work and tolerance
def _backbone_work(case, n):
    """Bytes that have to move (inputs, weights, output) and useful FLOPs of one forward on n points."""
    b = 2 if case["dtype"] == "bf16" else 4
    c_in = 6 if case["kind"] == "indoor" else 4
    per_scene = n / case["scenes"]
    ratio, near = POOLED[case["kind"]], NEIGHBOURS[case["kind"]]
    flops, weights = 2.0 * n * 25 * c_in * ENC_CHANNELS[0], 125.0 * c_in * ENC_CHANNELS[0]
    for depths, channels in ((ENC_DEPTHS, ENC_CHANNELS), (DEC_DEPTHS, DEC_CHANNELS)):
        for level, (depth, c) in enumerate(zip(depths, channels)):
            rows, keys = n * ratio ** level, min(1024.0, per_scene * ratio ** level)
            flops += depth * rows * (2.0 * (near + 13) * c * c + 4.0 * keys * c)
            weights += depth * (27.0 + 13.0) * c * c
    for level in range(4):
        rows = n * ratio ** level
        child = (DEC_CHANNELS + (ENC_CHANNELS[4],))[level + 1]
        flops += 2.0 * rows * ENC_CHANNELS[level] * (ENC_CHANNELS[level + 1] + DEC_CHANNELS[level])
        flops += 2.0 * rows * ratio * child * DEC_CHANNELS[level]
        weights += ENC_CHANNELS[level] * (ENC_CHANNELS[level + 1] + DEC_CHANNELS[level]) + child * DEC_CHANNELS[level]
    return n * (24.0 + b * c_in + b * DEC_CHANNELS[0]) + b * weights, flops


def work(case):
    path = case["path"]
    if path == "forward":
        n = case["scenes"] * case["size"] * (1.0 if case["kind"] == "indoor" else LIDAR_VOXELS)
        nbytes, flops = _backbone_work(case, n)
    elif path == "segment":
        n = case["scenes"] * case["size"]
        nbytes, flops = _backbone_work(case, n)
        # raw coordinates and features in; logits and row of every raw point out
        nbytes += n * RAW_PER_VOXEL * (12.0 + 12.0 + 2.0 * CLASSES + 8.0)
        flops += 2.0 * n * DEC_CHANNELS[0] * CLASSES
    elif path == "serialize":
        nbytes, flops = case["points"] * (12.0 + 4 * 24.0), 0.0
    elif path == "attention":
        n, c = case["points"], case["channels"]
        nbytes, flops = n * (4.0 * c + 8.0) + 8.0 * c * c, n * (8.0 * c * c + 4.0 * min(n, case["patch"]) * c)
    elif path == "xcpe":
        n, c = case["size"], case["channels"]
        nbytes, flops = n * (4.0 * c + 12.0) + 54.0 * c * c, 2.0 * n * NEIGHBOURS["indoor"] * c * c
    else:
        n = case["scenes"] * case["size"]
        # raw coordinates and features in, row of every raw point out; coordinates, cells and features of the voxels out
        nbytes, flops = n * RAW_PER_VOXEL * (12.0 + 24.0 + 8.0) + n * (12.0 + 12.0 + 24.0), 0.0
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    path = case["path"]
    if path in ("serialize", "voxelize"):
        return "exact"
    if case["dtype"] == "fp32":
        return {"rel": 5e-5}                    # 22 blocks of 32-bit sums
    if path in ("forward", "segment"):
        return {"rel": 2e-2, "max": 0.5}        # 22 blocks with bf16 activations
    return {"rel": 1e-2}
