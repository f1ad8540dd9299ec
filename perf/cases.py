"""Performance cases of the sparse 3D front end: what its users have it do, through the public entry points.

A case names one kind of call and its sizes. The listed ones come from the configurations of the benchmark and of the
tests: 20,000-point frames one at a time (the single-frame case and the real-time loop) and in batches, 120,000-point
frames (the throughput sweep), and the single layers that a plugin host calls one by one. `draw` spreads the same
kinds over the sizes between and around them.

Frames are drawn on the GPU with the distribution of the package's synth module: 65 % of the points on a ground sheet
whose density falls as 1/r^2 inside a sector, the rest inside car-sized boxes, rows in random order.
"""
import ctypes
import functools
import importlib.util
import math
import os
import sys

import torch

PACKAGE = "se_ssd_ai_trt_b200"
FULL_GRID = (41, 1600, 1408)


def package():
    """The package of the tree that is the working folder (its folder's name has dashes: it is loaded by path)."""
    if PACKAGE not in sys.modules:
        path = os.path.join(os.getcwd(), "se-ssd-ai-trt_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(PACKAGE, path, submodule_search_locations=[os.path.dirname(path)])
        sys.modules[PACKAGE] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[PACKAGE])
    return sys.modules[PACKAGE]


# ---- the cases -------------------------------------------------------------------------------------------------

def listed():
    return [
        # The voxeliser alone, on the frame of the single-frame configuration: the smallest call of the library.
        dict(name="voxelize 1 x 20k f32", kind="voxelize", frames=1, points=20000, half=False, ragged=False),
        # The same for frames that come in batches (offline preprocessing): the benchmark's voxelize workload.
        dict(name="voxelize 64 x 20k f32", kind="voxelize", frames=64, points=20000, half=False, ragged=False),
        # One submanifold layer as a plugin host calls it, fp32 as the reference runs it, on a full-resolution frame:
        # the benchmark's subm16 workload.
        dict(name="subm 16-16 f32 20k", kind="subm", level=0, cin=16, cout=16, frames=1, points=20000, half=False),
        # The same for a 64-channel layer in fp16 with its batch norm and ReLU, on the rows of a dense frame at 1/4
        # resolution.
        dict(name="subm 64-64 f16 120k", kind="subm", level=2, cin=64, cout=64, frames=1, points=120000, half=True),
        # A strided layer as a plugin host calls it: it makes new rows, and the host reads the status.
        dict(name="spconv 16-32 f16 20k", kind="spconv", level=0, cin=16, cout=32, frames=1, points=20000, half=True),
        # What follows the 2D head: decode, score filter, rotated NMS of one frame.
        dict(name="filter + nms 1", kind="post", frames=1, objects=25),
        # The whole front end, one 20,000-point frame at a time, in both feature types.
        dict(name="backbone 1 x 20k f16", kind="backbone", frames=1, points=20000, half=True, ragged=False),
        dict(name="backbone 1 x 20k f32", kind="backbone", frames=1, points=20000, half=False, ragged=False),
        # Several sensors' frames at once, each with its own number of points.
        dict(name="backbone 5 x 77k ragged f16", kind="backbone", frames=5, points=76543, half=True, ragged=True),
        # Frame to boxes with everything in one graph: the loop of a real-time detector.
        dict(name="detect 1 x 20k graph", kind="detect", points=20000),
        # Throughput on small frames that are already on the device, and on large ones that come from pinned host
        # memory (the benchmark's headline, which stands for recorded drives run through the network).
        dict(name="pipeline device 256 x 20k", kind="pipeline", frames=256, points=20000, batch=32, streams=4, host=False),
        dict(name="pipeline host 128 x 120k", kind="pipeline", frames=128, points=120000, batch=32, streams=2, host=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("voxelize", "subm", "spconv", "post", "backbone", "backbone", "detect", "pipeline"))
    if kind == "voxelize":
        points = _log_int(rng, 1000, 120000)
        return dict(kind=kind, frames=_log_int(rng, 1, max(1, min(64, 1500000 // points))), points=points,
                    half=rng.random() < 0.5, ragged=rng.random() < 0.5)
    if kind == "subm":
        level = rng.choice((0, 1, 2, 3))
        cin, cout = ((4, 16) if rng.random() < 0.5 else (16, 16)) if level == 0 else ((32, 32) if level == 1 else (64, 64))
        return dict(kind=kind, level=level, cin=cin, cout=cout, frames=rng.randint(1, 4), points=_log_int(rng, 3000, 120000),
                    half=rng.random() < 0.7)
    if kind == "spconv":
        level = rng.choice((0, 1, 2, 3))
        cin, cout = ((16, 32), (32, 64), (64, 64), (64, 64))[level]
        return dict(kind=kind, level=level, cin=cin, cout=cout, frames=rng.randint(1, 4), points=_log_int(rng, 3000, 120000),
                    half=rng.random() < 0.7)
    if kind == "post":
        return dict(kind=kind, frames=_log_int(rng, 1, 16), objects=rng.randint(3, 40))
    if kind == "backbone":
        half = rng.random() < 0.8
        points = _log_int(rng, 3000, 120000 if half else 40000)
        return dict(kind=kind, frames=rng.randint(1, 8 if half else 2), points=points, half=half, ragged=rng.random() < 0.5)
    if kind == "detect":
        return dict(kind=kind, points=_log_int(rng, 8000, 60000))
    points = _log_int(rng, 8000, 120000)
    batch, streams = rng.choice((8, 12, 16, 32)), rng.randint(2, 4)
    if points > 20000:
        streams = 2
    return dict(kind=kind, frames=rng.randint(batch * streams, 128), points=points, batch=batch, streams=streams,
                host=rng.random() < 0.6)


# ---- inputs ----------------------------------------------------------------------------------------------------

def lidar_frames(frames, points, seed, device="cuda"):
    """Frames [frames, points, 4] = (x, y, z, intensity) on the device, a function of the seed alone."""
    g = torch.Generator(device=device).manual_seed(seed * 2654435761 % (1 << 62))
    kw = dict(generator=g, device=device)
    boxes = 10 + round(points / 4000)                       # 15 at 20,000 points, 40 at 120,000
    # ground: radius by the inverse of its distribution, cut where the ray leaves the range
    az = (2.0 * torch.rand((frames, points), **kw) - 1.0) * math.radians(49.0)
    reach = torch.minimum(70.399 / torch.cos(az), 39.999 / torch.sin(az).abs().clamp_min(1e-6)).clamp_max(80.0)
    r = 1.0 / (0.5 - torch.rand((frames, points), **kw) * (0.5 - 1.0 / reach))
    gx, gy = r * torch.cos(az), r * torch.sin(az)
    gz = -1.7 + 0.05 * torch.randn((frames, points), **kw)
    # objects: 4 x 1.8 x 1.6 m boxes with random centres
    cx = 2.5 + torch.rand((frames, boxes), **kw) * 65.4
    cy = -38.5 + torch.rand((frames, boxes), **kw) * 77.0
    which = torch.randint(boxes, (frames, points), **kw)
    u = torch.rand((3, frames, points), **kw) - 0.5
    ox, oy, oz = cx.gather(1, which) + u[0] * 4.0, cy.gather(1, which) + u[1] * 1.8, -0.9 + u[2] * 1.6
    ground = torch.rand((frames, points), **kw) < 0.65
    out = torch.empty((frames, points, 4), device=device)
    out[..., 0] = torch.where(ground, gx, ox).clamp(0.0, 70.399)
    out[..., 1] = torch.where(ground, gy, oy).clamp(-40.0, 39.999)
    out[..., 2] = torch.where(ground, gz, oz).clamp(-2.999, 0.999)
    out[..., 3] = torch.rand((frames, points), **kw)
    return out


def frame_sizes(frames, points, ragged, seed):
    """Points of each frame: all of them, or any number from an eighth of them up."""
    if not ragged:
        return [points] * frames
    g = torch.Generator().manual_seed(seed + 17)
    return [int(v) for v in (points * (0.125 + 0.875 * torch.rand(frames, generator=g))).long().clamp(1, points)]


def max_voxels(points):
    """Row capacity that the frames of a size need at every level: the reference's constant for frames of its size,
    the benchmark's for larger ones."""
    return 60000 if points <= 20000 else 200000


def level_shape(level):
    return (FULL_GRID, (21, 800, 704), (11, 400, 352), (5, 200, 176))[level]


def level_rows(cloud, level):
    """Active cells [n, 3] = (z, y, x) of one frame at a level of the network: the frame's voxels, then per level the
    outputs that a 3x3x3 kernel of stride 2 makes of them. Voxels in random order (the voxeliser numbers them by their
    first point), derived rows in (z, y, x) order."""
    dev = cloud.device
    Z, Y, X = FULL_GRID
    low = torch.tensor([0.0, -40.0, -3.0], device=dev)
    size = torch.tensor([0.05, 0.05, 0.1], device=dev)
    x, y, z = ((cloud[:, :3] - low) / size).long().clamp_min(0).unbind(1)
    z, y, x = z.clamp_max(Z - 2), y.clamp_max(Y - 1), x.clamp_max(X - 1)
    key = torch.unique((z * Y + y) * X + x)
    if level == 0:
        g = torch.Generator(device=dev).manual_seed(int(key.sum()) % (1 << 40))
        key = key[torch.randperm(len(key), generator=g, device=dev)]
    for lv in range(1, level + 1):
        Zo, Yo, Xo = level_shape(lv)
        zyx = torch.stack((key // (Y * X), key // X % Y, key % X), 1)
        pad = torch.tensor([0 if lv == 3 else 1, 1, 1], device=dev)
        outs = []
        for d in range(8):
            o = torch.div(zyx + pad, 2, rounding_mode="floor") - torch.tensor([d >> 2 & 1, d >> 1 & 1, d & 1], device=dev)
            k = zyx - 2 * o + pad
            ok = ((k >= 0) & (k < 3) & (o >= 0) & (o < torch.tensor([Zo, Yo, Xo], device=dev))).all(1)
            o = o[ok]
            outs.append((o[:, 0] * Yo + o[:, 1]) * Xo + o[:, 2])
        key, (Z, Y, X) = torch.unique(torch.cat(outs)), (Zo, Yo, Xo)
    return torch.stack((key // (Y * X), key // X % Y, key % X), 1).int()


@functools.lru_cache(None)
def _network_weights():
    return package().random_weights()


@functools.lru_cache(None)
def _neck_weights():
    return package().detector.random_neck_weights()


def _backbone(points, half):
    pkg = package()
    w, scale, shift = _network_weights()
    return pkg.Backbone(max_voxels(points), w, scale, shift, dtype=pkg.F16 if half else pkg.F32)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](package(), case, seed)


def _points(case, seed):
    ragged = case.get("ragged", False)
    sizes = frame_sizes(case["frames"], case["points"], ragged, seed)
    return lidar_frames(case["frames"], case["points"], seed), torch.tensor(sizes, dtype=torch.int32, device="cuda")


def _prepare_voxelize(pkg, case, seed):
    B, P = case["frames"], case["points"]
    pts, sizes = _points(case, seed)
    params = pkg.voxel_params(20000 if P <= 20000 else 100000)
    V = params.max_voxels
    nbytes = pkg.lib().sessd_voxelize_workspace_bytes(ctypes.byref(params), B, P)
    return dict(kind="voxelize", pts=pts, sizes=sizes, params=params, dtype=pkg.F16 if case["half"] else pkg.F32,
                vox=torch.empty((B, V, 4), dtype=torch.float16 if case["half"] else torch.float32, device="cuda"),
                coors=torch.empty((B, V, 4), dtype=torch.int32, device="cuda"),
                num=torch.empty((B,), dtype=torch.int32, device="cuda"),
                ws=torch.empty(nbytes, dtype=torch.uint8, device="cuda"))


def _layer_inputs(pkg, case, seed):
    """Features, coordinates and row counts of a layer's input rows, and its weights with folded batch norm."""
    B, P, cin, cout, level = (case[k] for k in ("frames", "points", "cin", "cout", "level"))
    V, tdt = max_voxels(P), torch.float16 if case["half"] else torch.float32
    clouds = lidar_frames(B, P, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 3)
    feat = torch.zeros((B, V, cin), dtype=tdt, device="cuda")
    coors = torch.zeros((B, V, 4), dtype=torch.int32, device="cuda")
    num = []
    for b in range(B):
        rows = level_rows(clouds[b], level)[:V]
        n = len(rows)
        coors[b, :n, 0], coors[b, :n, 1:] = b, rows
        feat[b, :n] = torch.randn((n, cin), generator=g, device="cuda").relu_().to(tdt)   # rows come from a ReLU
        num.append(n)
    subm, shape = case["kind"] == "subm", level_shape(level)
    pad = (0, 1, 1) if level == 2 else (1, 1, 1)
    if subm:
        layer = pkg.schedule.ConvLayer("layer", True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), shape, shape)
    elif level == 3:
        layer = pkg.schedule.ConvLayer("layer", False, cin, cout, (3, 1, 1), (2, 1, 1), (0, 0, 0), shape, (2, 200, 176))
    else:
        layer = pkg.schedule.ConvLayer("layer", False, cin, cout, (3, 3, 3), (2, 2, 2), pad, shape, level_shape(level + 1))
    gw = torch.Generator().manual_seed(11 + 64 * level + cin)       # a network's weights do not change with its input
    w = (torch.randn((layer.kvol, cin, cout), generator=gw) / math.sqrt(layer.kvol * cin / 4)).numpy()
    scale = (1 + 0.1 * torch.randn(cout, generator=gw)).numpy()
    shift = (0.05 * torch.randn(cout, generator=gw)).numpy()
    params = pkg.conv_params(layer, V)
    weights = pkg.ConvWeights(params, w, scale, shift, True, pkg.F16 if case["half"] else pkg.F32)
    return feat, coors, torch.tensor(num, dtype=torch.int32, device="cuda"), params, weights


def _prepare_subm(pkg, case, seed):
    feat, coors, num, params, weights = _layer_inputs(pkg, case, seed)
    first = pkg.subm_conv(feat, coors, num, params, weights, keep_workspace=True)   # sizes the workspace and the output
    return dict(kind="subm", args=(feat, coors, num, params, weights), out=first["features"], ws=first["workspace"])


def _prepare_spconv(pkg, case, seed):
    return dict(kind="spconv", args=_layer_inputs(pkg, case, seed))


def _prepare_post(pkg, case, seed):
    B, (H, W) = case["frames"], (pkg.schedule.FEATURE_MAP_HEIGHT, pkg.schedule.FEATURE_MAP_WIDTH)
    g = torch.Generator(device="cuda").manual_seed(seed + 5)
    kw = dict(generator=g, device="cuda")
    # a head's output: low logits everywhere, and a patch of high ones around every object, for one of the two yaws
    logit = torch.randn((B, H, W, 2), **kw) * 0.5 - 5.0
    y = torch.arange(H, device="cuda").view(1, H, 1)
    x = torch.arange(W, device="cuda").view(1, 1, W)
    for _ in range(case["objects"]):
        cy, cx = (torch.rand((B, 1, 1), **kw) * n for n in (H, W))
        yaw = torch.randint(2, (B, 1, 1), **kw)
        bump = 8.0 * torch.exp(-((y - cy) ** 2 + (x - cx) ** 2) / 5.0)
        logit += bump[..., None] * torch.stack((yaw == 0, yaw == 1), -1)
    n = H * W * 2
    return dict(kind="post", box=0.1 * torch.randn((B, n, 7), **kw), cls=logit.reshape(B, n, 1).contiguous(),
                iou=(0.6 + 0.2 * torch.randn((B, n, 1), **kw)), dirs=torch.randn((B, n, 2), **kw),
                anchors=pkg.anchor_params(), filter=pkg.filter_params())


def _prepare_backbone(pkg, case, seed):
    bb = _backbone(case["points"], case["half"])
    pts, sizes = _points(case, seed)
    return dict(kind="backbone", bb=bb, pts=pts, sizes=sizes,
                ws=torch.empty(bb.workspace_bytes(case["frames"], case["points"]), dtype=torch.uint8, device="cuda"),
                dense=torch.empty(bb.dense_shape(case["frames"]), device="cuda",
                                  dtype=torch.float16 if case["half"] else torch.float32))


def _prepare_detect(pkg, case, seed):
    P = case["points"]
    pts, sizes = _points(dict(case, frames=1), seed)
    bb = _backbone(P, True)
    blobs = dict(_neck_weights())
    # random heads give outputs in the hundreds and pass half of their anchors: scaled to a trained head's range, and
    # with a classification bias that lets some 300 through
    heads = pkg.detector.Detector(bb, pkg.detector.Neck2D(blobs))(pts, sizes)["heads"]
    for name, std in (("box", 0.1), ("cls", 1.0), ("iou", 0.3), ("dir", 1.0)):
        factor = 2.0 ** round(math.log2(std / float(heads[name].std())))
        for part in (".weight", ".bias"):
            blobs["bbox_head.tasks.0.conv_" + name + part] = blobs["bbox_head.tasks.0.conv_" + name + part] * factor
        if name == "cls":
            threshold = pkg.schedule.SCORE_THRESHOLD
            lift = math.log(threshold / (1 - threshold)) - factor * float(torch.topk(heads[name].flatten(), 300).values[-1])
            blobs["bbox_head.tasks.0.conv_cls.bias"] = blobs["bbox_head.tasks.0.conv_cls.bias"] + lift
    det = pkg.detector.Detector(bb, pkg.detector.Neck2D(blobs)).capture(P)
    return dict(kind="detect", det=det, pts=pts.cpu().pin_memory(), sizes=sizes.cpu().pin_memory())


def _prepare_pipeline(pkg, case, seed):
    F, P = case["frames"], case["points"]
    bb = _backbone(P, True)
    pipe = pkg.Pipeline(bb, case["batch"], P, nstreams=case["streams"])
    pts, sizes = lidar_frames(F, P, seed), torch.full((F,), P, dtype=torch.int32, device="cuda")
    state = dict(kind="pipeline", bb=bb, pipe=pipe, host=case["host"], pts=pts, sizes=sizes)
    if case["host"]:
        for k in ("pts", "sizes"):
            state[k] = torch.empty(state[k].shape, dtype=state[k].dtype, pin_memory=True).copy_(state[k])
        state["num"], state["status"] = (torch.zeros((F,), dtype=torch.int32).pin_memory() for _ in range(2))
    # the maps that the slots hold after a run: those of the last group of each
    groups = -(-F // case["batch"])
    state["held"] = [(g % case["streams"], min(case["batch"], F - g * case["batch"]))
                     for g in range(max(0, groups - case["streams"]), groups)]
    return state


# ---- one pass --------------------------------------------------------------------------------------------------

def run(state):
    return globals()["_run_" + state["kind"]](package(), state)


def _run_voxelize(pkg, s):
    pkg.voxelize_into(s["pts"], s["sizes"], s["params"], s["vox"], s["coors"], s["num"], s["ws"], s["dtype"])
    return s["vox"], s["coors"], s["num"]


def _run_subm(pkg, s):
    pkg.subm_conv_into(*s["args"], s["out"], s["ws"])
    return s["out"]


def _run_spconv(pkg, s):
    r = pkg.sparse_conv(*s["args"])
    return r["features"], r["coors"], r["voxel_num"], r["status"]


def _run_post(pkg, s):
    f = pkg.filter_boxes(s["box"], s["cls"], s["iou"], s["dirs"], s["filter"], anchors=s["anchors"])
    kept, num = pkg.rotated_nms(f["box"], f["valid"])
    return kept, num, [f[k] for k in ("box", "score", "iou", "direction", "valid", "status")]


def _run_backbone(pkg, s):
    return s["bb"].run(s["pts"], s["sizes"], s["ws"], s["dense"])[0]


def _run_detect(pkg, s):
    out = s["det"].replay(s["pts"], s["sizes"])
    return out["boxes"], out["num"], out["status"], [out["heads"][k] for k in ("box", "cls", "iou", "dir")]


def _run_pipeline(pkg, s):
    counts = []
    if s["host"]:
        s["pipe"].run_host(s["pts"], s["sizes"], s["num"], s["status"])
        counts = [s["num"], s["status"]]
    else:
        s["pipe"].run_device(s["pts"], s["sizes"])
    maps = [s["pipe"].dense(slot)[:n] for slot, n in s["held"]]
    for m in maps:
        m.pipeline = s["pipe"]         # the maps are the pipeline's own memory: it lives as long as they do
    return counts, maps


# ---- what a pass cannot do without -----------------------------------------------------------------------------

MAP_VALUES = 128 * 200 * 176          # of one frame's dense BEV map


def _rows(points, level):
    """Rows of a frame of so many points at a level (0 .. 3), fitted to the frames above."""
    at20k, at120k = ((17450, 82500), (38200, 160000), (26300, 77500), (11200, 28500))[level]
    return at20k * (points / 20000) ** (math.log(at120k / at20k) / math.log(6.0))


def _pairs(points, level):
    """Rulebook pairs per frame of a submanifold layer of a level (0 .. 3), fitted likewise."""
    at20k, at120k = ((68000, 405000), (364000, 2000000), (417000, 1300000), (156000, 430000))[level]
    return at20k * (points / 20000) ** (math.log(at120k / at20k) / math.log(6.0))


def _strided_pairs(points, level):
    """The same for the strided layer that leaves a level."""
    return (3.4, 3.4, 3.4, 1.2)[level] * _rows(points, level)


def _backbone_flops(points):
    subm = (4 * 16 + 16 * 16, 2 * 32 * 32, 3 * 64 * 64, 3 * 64 * 64)
    strided = (16 * 32, 32 * 64, 64 * 64, 64 * 64)
    return 2.0 * sum(_pairs(points, lv) * subm[lv] + _strided_pairs(points, lv) * strided[lv] for lv in range(4))


def work(case):
    kind, P, F = case["kind"], case.get("points", 0), case.get("frames", 1)
    e = 2 if case.get("half", True) else 4
    if case.get("ragged"):
        P = P * 9 // 16                # the mean of the sizes
    if kind == "voxelize":
        V = 20000 if case["points"] <= 20000 else 100000
        return dict(bytes=F * (16 * P + V * (4 * e + 16) + 4), flops=F * 20 * P)
    if kind in ("subm", "spconv"):
        lv, cin, cout, V = case["level"], case["cin"], case["cout"], max_voxels(P)
        kvol = 3 if kind == "spconv" and lv == 3 else 27
        pairs = _pairs(P, lv) if kind == "subm" else _strided_pairs(P, lv)
        out = V * cout * e + (V * 16 if kind == "spconv" else 0)      # outputs are whole: rows past the count are zeros
        return dict(bytes=F * (_rows(P, lv) * (cin * e + 16) + out) + kvol * cin * cout * e, flops=2.0 * F * pairs * cin * cout)
    if kind == "post":
        # every logit; the other head outputs only of the anchors that pass
        return dict(bytes=F * (70400 * 4 + 500 * (7 + 1 + 2 + 12 + 9) * 4), flops=F * 70400 * 10)
    weights = 2 * 10 ** 6 // 4 * e
    if kind == "backbone":
        return dict(bytes=F * (16 * P + MAP_VALUES * e) + weights, flops=F * _backbone_flops(P))
    if kind == "detect":
        # the 2D neck and head: 14 dense convolutions, 91 GFLOP; their outputs in fp32
        return dict(bytes=16 * P + 70400 * 11 * 4 + weights + 6 * 10 ** 6, flops=_backbone_flops(P) + 9.1e10)
    return dict(bytes=F * (16 * P + MAP_VALUES * e) + weights, flops=F * _backbone_flops(P))


def tolerance(case):
    kind = case["kind"]
    if kind == "voxelize":
        return {"rel": 1e-3} if case["half"] else {"rel": 1e-6}      # the mean of five values; rows and counts exactly
    if kind == "post":
        return {"rel": 1e-5}
    if not case.get("half", True):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-2} if kind in ("backbone", "pipeline", "detect") else {"rel": 2e-3}
