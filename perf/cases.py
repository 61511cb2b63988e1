"""The calls a program makes through this package, at the sizes it makes them: what a change of the kernels is timed on.

`listed()` names twelve of them, `draw()` gives more of the same kinds.  Three groups:

* whole frames (`op = "frame"`): points in, BEV map and kept boxes (detection) or per-point logits (segmentation) out,
  by the pipeline objects captured in a CUDA graph, the way a vehicle or an annotation server runs them.
  `mode = "shared"` is the pipelines' default; `mode = "engine"` is what an inference engine built from an exported
  graph executes: one stream, every node through its plugin entry point.
* single operators and the short chains they come in (`op` = "subm", "down_up", "mean_encoder", "cylinder", "head",
  "nms", "densify"), called through `deploy3d_b200.ops`; the operators whose number of output rows depends on the
  data (encoders, strided rulebooks) as plugin objects that write into buffers sized once per model.
* among these the small calls (a few hundred boxes, a few thousand voxels), where launches and the host path decide.

Data is synthetic and made on the GPU from the seed: a ground plane whose density falls off with the range plus
object-like clusters, in random order, as the package's own benchmark inputs.
"""
import math

import numpy as np
import torch

from deploy3d_b200 import ops
from deploy3d_b200.pipeline import DetectionPipeline, SegmentationPipeline
from deploy3d_b200.plugins import deserialize_plugin

DEV = "cuda:0"
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
ESIZE = {"fp32": 4, "fp16": 2, "bf16": 2}
CALIBRATION_SEED = 4711  # the frame buffer sizes are fixed with, once per model

# point cloud ranges and grids of the frame pipelines: x, y, z range; columns of a point
NETS = {"centerpoint": dict(rng=((-54, 54), (-54, 54), (-5, 3)), cols=5),
        "second": dict(rng=((0, 70.4), (-40, 40), (-3, 1)), cols=4),
        "cylinder3d": dict(rng=((-50, 50), (-50, 50), (-4, 2)), cols=4)}
GRID = (41, 1600, 1408)  # Z, Y, X of the voxel grid the single-operator rulebooks work on
# submanifold layers: the grid a backbone has reached when its features are this wide
GRID_OF = {16: GRID, 32: (21, 800, 704), 64: (11, 400, 352), 128: (8, 200, 176)}


def listed():
    return [
        # small: the boxes of one sweep of a three-class head after a score threshold
        dict(name="nms_3x257", op="nms", rows=3, boxes=257),
        # a detection head: per class top-500 of a 180 x 180 map, decoded, then rotated NMS; two scans per batch
        dict(name="head_180x180_fp16", op="head", batch=2, classes=3, size=180, topk=500, dtype="fp16"),
        # one 10-sweep cloud into voxels
        dict(name="mean_encoder_300k", op="mean_encoder", points=299993, cols=5),
        # point <-> voxel half of a segmentation network: cylinder voxels, per-voxel max, gathered back to the points
        dict(name="cylinder_points_120k", op="cylinder", points=120000, mean=False),
        # sparse -> dense hand-over to a 2-D head: 2 x 200 x 176 cells, 128 channels
        dict(name="densify_31k_fp16", op="densify", voxels=31337, channels=128, dtype="fp16"),
        # one fp32 submanifold layer over a sparse cloud
        dict(name="subm_20k_16_fp32", op="subm", voxels=20000, cin=16, cout=16, layers=1, dtype="fp32"),
        # a residual block at the deep, wide end of a backbone: rulebook and two layers over it
        dict(name="subm_66k_128_bf16", op="subm", voxels=66001, cin=128, cout=128, layers=2, dtype="bf16"),
        # strided convolution and its inverse (encoder-decoder), two scans per batch
        dict(name="down_up_120k_32_64_fp16", op="down_up", voxels=120000, cin=32, cout=64, dtype="fp16"),
        # single-sweep detection, bf16
        dict(name="frame_second_120k_bf16", op="frame", net="second", points=120000, dtype="bf16", mode="shared"),
        # 10-sweep detection, the largest detector
        dict(name="frame_centerpoint_300k", op="frame", net="centerpoint", points=300000, dtype="fp16", mode="shared"),
        # the same detector node by node, as an inference engine runs the exported graph
        dict(name="engine_centerpoint_300k", op="frame", net="centerpoint", points=300000, dtype="fp16",
             mode="engine"),
        # point-wise segmentation of one scan
        dict(name="frame_cylinder3d_120k", op="frame", net="cylinder3d", points=120000, dtype="fp16", mode="shared"),
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, spread evenly over its logarithm, odd as often as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["nms", "head", "mean_encoder", "cylinder", "densify", "subm", "down_up", "frame"])
    half = rng.choice(["fp16", "bf16"])
    if op == "nms":
        return dict(op=op, rows=rng.randint(1, 10), boxes=_spread(rng, 64, 1000))
    if op == "head":
        return dict(op=op, batch=rng.randint(1, 2), classes=rng.randint(1, 3), size=rng.randint(64, 256),
                    topk=_spread(rng, 50, 1000), dtype=rng.choice(["fp16", "fp32"]))
    if op == "mean_encoder":
        return dict(op=op, points=_spread(rng, 2000, 480000), cols=rng.choice([4, 5]))
    if op == "cylinder":
        return dict(op=op, points=_spread(rng, 2000, 480000), mean=rng.random() < 0.3)
    if op == "densify":
        return dict(op=op, voxels=_spread(rng, 500, 60000), channels=rng.choice([64, 128]),
                    dtype=rng.choice(["fp16", "bf16", "fp32"]))
    if op == "subm":
        if rng.random() < 0.3:
            c = rng.choice([16, 32])
            return dict(op=op, voxels=_spread(rng, 1000, 60000), cin=c, cout=c, layers=1, dtype="fp32")
        c = rng.choice([16, 32, 64, 128])
        return dict(op=op, voxels=_spread(rng, 1000, 100000 if c == 128 else 200000), cin=c, cout=c, layers=2,
                    dtype=half)
    if op == "down_up":
        c = rng.choice([16, 32, 64])
        return dict(op=op, voxels=_spread(rng, 2000, 200000), cin=c, cout=2 * c, dtype=half)
    net = rng.choice(["centerpoint", "second", "cylinder3d"])
    mode = "engine" if net != "cylinder3d" and rng.random() < 0.3 else "shared"
    return dict(op=op, net=net, points=_spread(rng, 20000, 300000 if net == "centerpoint" else 120000), dtype=half,
                mode=mode)


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _u(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device=DEV) * (hi - lo) + lo


def _points(g, n, ranges, cols):
    """n points [x, y, z, intensity (, time of one of ten sweeps)]: 70 % ground, density ~ 1 / r, 30 % clusters."""
    (x0, x1), (y0, y1), (z0, z1) = ranges
    rmax = max(abs(x0), abs(x1), abs(y0), abs(y1))
    got = []
    have = 0
    while have < n:
        need = int((n - have) * 3) + 256
        ng = int(need * 0.7)
        r, th = _u(g, ng, 2.0, rmax * 1.2), _u(g, ng, 0, 2 * math.pi)
        ground = torch.stack([r * th.cos(), r * th.sin(),
                              -1.7 + 0.08 * torch.randn(ng, generator=g, device=DEV)], 1)
        centres = torch.stack([_u(g, 40, x0, x1), _u(g, 40, y0, y1), _u(g, 40, -1.7, -0.2)], 1)
        nc = need - ng
        which = torch.randint(0, 40, (nc,), generator=g, device=DEV)
        clus = centres[which] + torch.randn((nc, 3), generator=g, device=DEV) * torch.tensor([0.9, 0.9, 0.5], device=DEV)
        p = torch.cat([ground, clus])
        p = p[(p[:, 0] > x0) & (p[:, 0] < x1) & (p[:, 1] > y0) & (p[:, 1] < y1) & (p[:, 2] > z0) & (p[:, 2] < z1)]
        got.append(p[torch.randperm(p.shape[0], generator=g, device=DEV)])
        have += p.shape[0]
    p = torch.cat(got)[:n]
    extra = [_u(g, n).unsqueeze(1)]
    if cols == 5:
        extra.append(torch.randint(0, 10, (n, 1), generator=g, device=DEV) * 0.05)
    return torch.cat([p] + extra, 1).contiguous()


def _voxels(g, n, grid, batch=1):
    """n distinct voxels [b, z, y, x], spread like the points, in random order."""
    z, y, x = grid
    cy, cx, rmax = y / 2.0, x / 2.0, min(y, x) / 2.0 - 1
    keys = torch.empty(0, dtype=torch.int64, device=DEV)
    while keys.numel() < n:
        need = int((n - keys.numel()) * 1.3) + 64
        ng = int(need * 0.7)
        r, th = _u(g, ng, 1.0, rmax), _u(g, ng, 0, 2 * math.pi)
        ground = torch.stack([torch.randint(0, min(4, z), (ng,), generator=g, device=DEV).float(), cy + r * th.sin(),
                              cx + r * th.cos()], 1)
        nc = need - ng
        centres = torch.stack([_u(g, 40, 0, z), _u(g, 40, 0, y), _u(g, 40, 0, x)], 1)
        which = torch.randint(0, 40, (nc,), generator=g, device=DEV)
        clus = centres[which] + torch.randn((nc, 3), generator=g, device=DEV) * torch.tensor([2.0, 8.0, 8.0],
                                                                                           device=DEV)
        v = torch.cat([ground, clus]).floor().long()
        b = torch.randint(0, batch, (need,), generator=g, device=DEV)
        zz, yy, xx = v[:, 0].clamp(0, z - 1), v[:, 1].clamp(0, y - 1), v[:, 2].clamp(0, x - 1)
        keys = torch.unique(torch.cat([keys, ((b * z + zz) * y + yy) * x + xx]))
    keys = keys[torch.randperm(keys.numel(), generator=g, device=DEV)[:n]]
    out = torch.stack([keys // (z * y * x), keys // (y * x) % z, keys // x % y, keys % x], 1)
    return out.to(torch.int32).contiguous()


def _boxes(g, rows, k):
    """Candidate boxes of `rows` classes, scores descending; a third of them crowd around object centres."""
    xy = _u(g, rows * k * 2, -54, 54).view(rows, k, 2)
    centres = _u(g, rows * 20 * 2, -50, 50).view(rows, 20, 2)
    which = torch.randint(0, 20, (rows, k), generator=g, device=DEV)
    near = centres.gather(1, which.unsqueeze(-1).expand(-1, -1, 2)) + 0.8 * torch.randn((rows, k, 2), generator=g,
                                                                                       device=DEV)
    xy = torch.where((_u(g, rows * k).view(rows, k, 1) < 0.33), near, xy)
    rest = torch.stack([_u(g, rows * k, -5, 3), _u(g, rows * k, 0.5, 5), _u(g, rows * k, 0.5, 5),
                        _u(g, rows * k, 0.5, 5), _u(g, rows * k, -math.pi, math.pi)], 1).view(rows, k, 5)
    scores = torch.sort(_u(g, rows * k).view(rows, k), dim=1, descending=True).values
    return scores.contiguous(), torch.cat([xy, rest], 2).contiguous()


def _weight(seed, kvol, cin, cout):
    r = np.random.Generator(np.random.PCG64(int(seed)))
    w = (r.standard_normal((kvol, cin, cout)) * math.sqrt(2.0 / (kvol * cin))).astype(np.float32)
    return w, (0.05 * r.standard_normal(cout)).astype(np.float32)


def _int(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _shape(dims):
    return torch.empty(dims, dtype=torch.int32, device=DEV)


_SIZES = {}  # buffer sizes of a model, fixed once from a calibration frame, as an engine's are


def _sized(case, measure):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _SIZES:
        _SIZES[key] = measure()
    return _SIZES[key]


def _roomy(count):
    return (int(count * 1.15) + 256 + 1023) // 1024 * 1024


# ---- one kind after the other ---------------------------------------------------------------------------------------
def _frame_pipe(case, caps):
    dt = DTYPES[case["dtype"]]
    if case["net"] == "cylinder3d":
        return SegmentationPipeline(DEV, n_pts=case["points"], dtype=dt, caps=caps)
    return DetectionPipeline(case["net"], DEV, n_pts=case["points"], dtype=dt, caps=caps,
                             plugin_order=case["mode"] == "engine")


def _calibrated(case):
    """Voxel buffers with 15 % of room over a calibration frame's counts."""
    n, net = case["points"], NETS[case["net"]]
    seg = case["net"] == "cylinder3d"
    roomy = None if seg else {"in": n, "down2": 5 * n, "down3": 5 * n, "down4": 4 * n, "out": 4 * n}
    pipe = _frame_pipe(case, roomy)
    if seg:
        pipe = _frame_pipe(case, {k: (n if k == "in" else 3 * n) for k in pipe.set_names})
    pipe.points.copy_(_points(_gen(CALIBRATION_SEED), n, net["rng"], net["cols"]))
    pipe.enqueue()
    counts = dict(pipe.net.counts())
    counts["in"] = int(pipe.vox_num.item())
    return {k: min(_roomy(v), n) if k == "in" else _roomy(v) for k, v in counts.items()}


def _prepare_frame(case, g):
    caps = dict(_sized(case, lambda: _calibrated(case)))
    net = NETS[case["net"]]
    s = dict(pipe=_frame_pipe(case, caps), points=_points(g, case["points"], net["rng"], net["cols"]))
    if case["net"] != "cylinder3d":
        s["scores"], s["boxes"] = _boxes(g, 10, 1000)
        s["pipe"].scores.copy_(s["scores"])
        s["pipe"].boxes.copy_(s["boxes"])
    s["pipe"].points.copy_(s["points"])
    s["pipe"].capture()
    return s


def _run_frame(s):
    pipe = s["pipe"]
    pipe.points.copy_(s["points"])  # the frame that just arrived
    if "scores" not in s:
        pipe.replay()
        return dict(logits=pipe.logits, labels=pipe.labels, voxels=pipe.vox_num)
    pipe.scores.copy_(s["scores"])
    pipe.boxes.copy_(s["boxes"])
    pipe.replay()
    return dict(bev=pipe.bev, scores=pipe.nms_scores, voxels=pipe.vox_num)


def _prepare_subm(case, g):
    n, c, dt = case["voxels"], case["cin"], DTYPES[case["dtype"]]
    grid = GRID_OF[c]
    s = dict(coors=_voxels(g, n, grid), num=_int([n]), shape=_shape([1, 0, *grid]), n=n, cin=c, cout=case["cout"])
    s["feats"] = torch.randn((n, c), generator=g, device=DEV).to(dt)
    s["layers"] = [_weight(17 + i, 27, c if i == 0 else case["cout"], case["cout"]) for i in range(case["layers"])]
    return s


def _run_subm(s):
    one = (1, 1, 1)
    index, num_index = ops.spconv_index(s["coors"], s["num"], s["shape"], (3, 3, 3), one, one, one, (0, 0, 0), s["n"],
                                        True, False)
    x, cin = s["feats"], s["cin"]
    for w, b in s["layers"]:
        x = torch.relu_(ops.spconv_mm(x, s["num"], s["num"], index, num_index, (3, 3, 3), cin, s["cout"], s["n"], True,
                                      False, w, b))
        cin = s["cout"]
    return dict(feats=x, index=index, num_index=num_index)


def _down(s):
    return s["rulebook"].enqueue(s["coors"], s["num"], s["shape"], outputs=s["buffers"])


def _prepare_down_up(case, g):
    n, dt, kvol = case["voxels"], DTYPES[case["dtype"]], 27

    def make(gen, max_out):
        half = [2, 0] + [(v + 1) // 2 for v in GRID]
        return dict(coors=_voxels(gen, n, GRID, batch=2), num=_int([n]), shape=_shape([2, 0, *GRID]), n=n,
                    max_out=max_out,
                    rulebook=deserialize_plugin("SPConvIdx3d", ops.data_s_spconv_index(
                        (3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1), (0, 0, 0), max_out, False, False)),
                    buffers=[_shape([3, kvol * (n + 128)]), _int([0]),
                             torch.zeros((max_out, 4), dtype=torch.int32, device=DEV), _int([0]), _shape(half)])

    max_out = _sized(case, lambda: _roomy(int(_down(make(_gen(CALIBRATION_SEED), 8 * n))[3].item())))
    s = make(g, max_out)
    s.update(cin=case["cin"], cout=case["cout"])
    s["feats"] = torch.randn((n, case["cin"]), generator=g, device=DEV).to(dt)
    s["w_down"], s["w_up"] = _weight(5, kvol, case["cin"], case["cout"]), _weight(6, kvol, case["cout"], case["cin"])
    return s


def _run_down_up(s):
    index, num_index, coors, num_out, _ = _down(s)
    ks = (3, 3, 3)
    mid = torch.relu_(ops.spconv_mm(s["feats"], s["num"], num_out, index, num_index, ks, s["cin"], s["cout"],
                                    s["max_out"], False, False, *s["w_down"]))
    up = ops.spconv_mm(mid, num_out, s["num"], index, num_index, ks, s["cout"], s["cin"], s["n"], False, True,
                       *s["w_up"])
    return dict(up=up, mid=mid, coors=coors, num_out=num_out, index=index, num_index=num_index)


MEAN_CFG = {5: ([-54, -54, -5, 0.075, 0.075, 0.2], [1, 0, 41, 1440, 1440], "centerpoint"),
            4: ([0, -40, -3, 0.05, 0.05, 0.1], [1, 0, 41, 1600, 1408], "second")}


def _prepare_mean_encoder(case, g):
    cfg, shape, net = MEAN_CFG[case["cols"]]
    n, c = case["points"], case["cols"]
    return dict(points=_points(g, n, NETS[net]["rng"], c), batch=_int([0]).repeat(n),
                cfg=torch.tensor(cfg, dtype=torch.float32, device=DEV), shape=_shape(shape),
                encoder=deserialize_plugin("SimpleMeanEncoder", ops.data_s_voxel_encoder(n)),
                buffers=[torch.zeros((n, c), device=DEV), _int([0]).repeat(n * 4).view(n, 4), _int([0])])


def _run_mean_encoder(s):
    feats, coors, num = s["encoder"].enqueue(s["points"], s["batch"], s["cfg"], s["shape"], outputs=s["buffers"])
    return dict(feats=feats, coors=coors, num=num)


def _prepare_cylinder(case, g):
    n = case["points"]
    return dict(points=_points(g, n, NETS["cylinder3d"]["rng"], 4), batch=_int([0]).repeat(n),
                cfg=torch.tensor([-4, -math.pi, 0, 2, math.pi, 50], dtype=torch.float32, device=DEV),
                shape=_shape([1, 0, 480, 360, 32]), reduce=1 if case["mean"] else 0,
                encoder=deserialize_plugin("CylinderEncoder", ops.data_s_voxel_encoder(n)),
                buffers=[torch.zeros((n, 9), device=DEV), _int([0]).repeat(n), _int([0]).repeat(n),
                         _int([0]).repeat(n * 4).view(n, 4), _int([0])])


def _run_cylinder(s):
    pts, to, count, coors, num = s["encoder"].enqueue(s["points"], s["batch"], s["cfg"], s["shape"],
                                                      outputs=s["buffers"])
    voxels = ops.scatter_to(pts, to, count, s["reduce"])
    back = ops.gather_back(voxels, to, 0.0)
    return dict(points=pts, to=to, count=count, coors=coors, num=num, voxels=voxels, back=back)


def _prepare_head(case, g):
    b, c, n, dt = case["batch"], case["classes"], case["size"], DTYPES[case["dtype"]]
    # class scores: a low background and a few hundred peaks
    scores = torch.rand((b, c, n, n), generator=g, device=DEV) ** 4 * 0.6
    scores = torch.where(torch.rand((b, c, n, n), generator=g, device=DEV) < 0.01,
                         torch.rand((b, c, n, n), generator=g, device=DEV), scores)
    ang = _u(g, b * n * n, -math.pi, math.pi).view(b, n, n)
    pred = torch.cat([torch.rand((b, 2, n, n), generator=g, device=DEV),
                      torch.rand((b, 1, n, n), generator=g, device=DEV) * 4 - 3,
                      torch.rand((b, 3, n, n), generator=g, device=DEV) * 2.5 - 1, ang.unsqueeze(1) * 1.2,
                      ang.sin().unsqueeze(1), ang.cos().unsqueeze(1)], 1)
    return dict(scores=scores.to(dt).contiguous(), pred=pred.to(dt).contiguous(), classes=tuple(range(c)),
                topk=case["topk"], cfg=torch.tensor([-54, -54, -5, 0.075, 0.075, 0.2], device=DEV))


def _run_head(s):
    out = ops.yolox3d_decode(s["scores"], s["pred"], s["cfg"], 8, s["classes"], s["topk"])
    kept = [ops.nms3d(out[3 * i + 1], out[3 * i + 2], 0.2) for i in range(len(s["classes"]))]
    return dict(decoded=list(out), kept=kept)


def _prepare_nms(case, g):
    scores, boxes = _boxes(g, case["rows"], case["boxes"])
    return dict(scores=scores, boxes=boxes)


def _run_nms(s):
    return ops.nms3d(s["scores"], s["boxes"], 0.2)


def _prepare_densify(case, g):
    n, c = case["voxels"], case["channels"]
    coors = _voxels(g, n, (2, 200, 176))
    feats = torch.relu(torch.randn((n, c), generator=g, device=DEV)).to(DTYPES[case["dtype"]])
    return dict(feats=feats, coors=coors, num=_int([n]), shape=_shape([1, 0, 2, 200, 176]), channels=2 * c)


def _run_densify(s):
    return ops.bev_densify(s["feats"], s["coors"], s["num"], s["shape"], s["channels"])


_KINDS = {"frame": (_prepare_frame, _run_frame), "subm": (_prepare_subm, _run_subm),
          "down_up": (_prepare_down_up, _run_down_up), "mean_encoder": (_prepare_mean_encoder, _run_mean_encoder),
          "cylinder": (_prepare_cylinder, _run_cylinder), "head": (_prepare_head, _run_head),
          "nms": (_prepare_nms, _run_nms), "densify": (_prepare_densify, _run_densify)}


def prepare(case, seed):
    state = _KINDS[case["op"]][0](case, _gen(seed))
    state["op"] = case["op"]
    return state


def run(state):
    return _KINDS[state["op"]][1](state)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
# Layers of a frame's network: voxels per point and pairs (input, offset) per output voxel as counted on a frame of
# `full` points and on one of a quarter of them (in between and beyond: along the logarithm), layers alike, cin, cout,
# kernel volume.  A set's features are counted once written and once read between two layers.
_LAYERS = {
    "centerpoint": (300000, [
        (0.94, 0.98, 3.0, 1.6, 5, 16, 16, 27), (1.55, 2.30, 1.8, 1.25, 1, 16, 32, 27),
        (1.55, 2.30, 11.5, 8.5, 4, 32, 32, 27), (0.80, 1.74, 5.7, 3.85, 1, 32, 64, 27),
        (0.80, 1.74, 16.3, 12.3, 4, 64, 64, 27), (0.22, 0.85, 12.5, 7.7, 1, 64, 128, 27),
        (0.22, 0.85, 18.3, 17.9, 4, 128, 128, 27), (0.21, 0.81, 1.6, 1.55, 1, 128, 128, 3)]),
    "second": (120000, [
        (0.99, 1.00, 1.5, 1.1, 2, 16, 16, 27), (2.70, 3.17, 1.2, 1.06, 1, 16, 32, 27),
        (2.70, 3.17, 10.2, 6.7, 2, 32, 32, 27), (1.91, 3.28, 4.6, 3.2, 1, 32, 64, 27),
        (1.91, 3.28, 15.8, 12.9, 2, 64, 64, 27), (0.75, 1.81, 8.4, 5.9, 1, 64, 64, 27),
        (0.75, 1.81, 18.9, 15.5, 2, 64, 64, 27), (0.54, 1.42, 1.85, 1.7, 1, 64, 128, 3)]),
    "cylinder3d": (120000, [
        (0.74, 0.83, 2.46, 1.5, 4, 32, 32, 9), (0.74, 0.83, 2.46, 1.5, 4, 56, 64, 9),
        (0.74, 1.56, 3.05, 1.6, 1, 64, 64, 27), (0.74, 1.56, 5.75, 4.4, 4, 112, 128, 9),
        (0.25, 0.77, 9.6, 6.1, 1, 128, 128, 27), (0.25, 0.77, 6.7, 6.0, 4, 224, 256, 9),
        (0.12, 0.44, 14.3, 11.8, 1, 256, 256, 27), (0.12, 0.44, 22.7, 22.3, 1, 256, 256, 27),
        (0.25, 0.77, 6.6, 6.7, 1, 256, 256, 27), (0.25, 0.77, 6.7, 6.0, 2, 256, 256, 9),
        (0.25, 0.77, 19.7, 17.4, 1, 256, 256, 27), (0.25, 0.77, 19.7, 17.4, 1, 256, 128, 27),
        (0.74, 1.56, 3.3, 3.0, 1, 128, 128, 27), (0.74, 1.56, 5.75, 4.4, 2, 128, 128, 9),
        (0.74, 1.56, 16.5, 11.4, 1, 128, 128, 27), (0.74, 1.56, 16.5, 11.4, 1, 128, 64, 27),
        (0.74, 0.83, 3.07, 3.06, 1, 64, 64, 27), (0.74, 0.83, 2.46, 1.5, 2, 64, 64, 9),
        (0.74, 0.83, 5.8, 2.6, 1, 64, 64, 27), (0.74, 0.83, 1.45, 1.15, 3, 64, 64, 3),
        (0.74, 0.83, 5.8, 2.6, 1, 128, 20, 27)])}


def work(case):
    op, e = case["op"], ESIZE.get(case.get("dtype"), 4)
    if op == "frame":
        n = case["points"]
        full, rows = _LAYERS[case["net"]]
        t = math.log(full / n) / math.log(4.0)  # 0 at the full size, 1 at a quarter of it
        flops = feats = weights = 0.0
        for v0, v1, p0, p1, layers, a, b, kvol in rows:
            m, p = n * v0 * (v1 / v0) ** t, p0 * (p1 / p0) ** t
            flops += 2.0 * m * p * layers * a * b
            feats += m * e * layers * (a + b)
            weights += kvol * a * b * e * layers
        if case["net"] == "cylinder3d":
            return dict(bytes=feats + weights + n * (16 + 4 + 4 * 20 + 4), flops=flops)
        bev = 256 * (180 * 180 if case["net"] == "centerpoint" else 200 * 176) * e
        return dict(bytes=feats + weights + n * (4 * NETS[case["net"]]["cols"] + 4) + bev + 10 * 1000 * 36,
                    flops=flops)
    if op == "subm":
        n, c, l = case["voxels"], case["cin"], case["layers"]
        # neighbours a voxel has of 27 (itself one of them), on the fine grid of the narrow layers and on coarser ones
        pairs = n * min(20.0, 1 + {16: 0.9, 32: 1.56, 64: 3.6, 128: 10.0}[c] * (n / 66000.0) ** 0.8)
        return dict(bytes=16 * n + 12 * 27 * (n + 128) + l * (2 * n * c * e + 27 * c * c * e),
                    flops=2 * pairs * c * c * l)
    if op == "down_up":
        n, a, b = case["voxels"], case["cin"], case["cout"]
        m, pairs = 2.8 * n, 3.36 * n
        return dict(bytes=16 * (n + m) + 12 * 27 * (n + 128) + e * (2 * n * a + 2 * m * b) + 2 * 27 * a * b * e,
                    flops=4 * pairs * a * b)
    if op == "mean_encoder":
        n, c = case["points"], case["cols"]
        return dict(bytes=n * (4 * c + 4) + n * 4 * c + 0.9 * n * 16, flops=2.0 * n * c)
    if op == "cylinder":
        n, m = case["points"], 0.7 * case["points"]
        # points in; 9 columns per point, voxel id, point counts, coordinates out; voxel features and point rows out
        return dict(bytes=n * 20 + n * 40 + 4 * n + 16 * m + 36 * n + 36 * n, flops=30.0 * n)
    if op == "head":
        b, c, n, k = case["batch"], case["classes"], case["size"] ** 2, case["topk"]
        return dict(bytes=b * c * (n * e + k * (9 * e + 4 + 4 + 28 + 4)), flops=b * c * (n + k * k / 2 * 12.0))
    if op == "nms":
        r, k = case["rows"], case["boxes"]
        return dict(bytes=r * k * 36, flops=r * k * k / 2 * 12.0)
    n, c = case["voxels"], case["channels"]
    return dict(bytes=n * (c * e + 16) + 2 * 200 * 176 * c * e, flops=1.0 * n * c)


def tolerance(case):
    op = case["op"]
    if op == "frame":  # a dozen to forty layers that round to 16 bits each; argmax labels may tie
        return {"rel": 5e-3 if case["dtype"] == "fp16" else 2e-2, "differ": 5e-3}
    if op in ("subm", "down_up"):  # fp32 sums; one or two roundings to 16 bits on the way
        return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
    if op in ("mean_encoder", "cylinder", "head"):  # 32-bit sums in any order; expf / atan2f of single cells
        return {"rel": 1e-5}
    return "exact"
