"""What a program that uses this package has it do, as cases that can be timed.

Seven kinds of work, each through the public entry points:

infer    set-abstraction stack of a point network, forward only: sampling and fused grouping per
         level; with ``decoder`` the interpolation back up as well (segmentation)
train    the same stack with three_nn / three_interpolate, forward and backward; the grouping either
         as separate calls (ball_query, grouping_operation) or fused (sa_group)
search   dense ball query and kNN of a batch, and the three-neighbour interpolation back
packed   ball query and kNN over a ragged batch of scenes (partial_dense layout)
chamfer  Chamfer loss of a batch of pairs and its gradient, for one cloud of a pair or both
cloud    sampling and ball query of large scans
segment  instance segmentation: region growing of the predicted classes, IoU with the ground truth
grnet    gridding and cubic feature sampling of a completion network, forward and backward

A case is a dict of plain values; sizes inside a case that have to be ragged follow from it by a
fixed rule, values follow from the seed.
"""
import math

import torch

import torch_points_kernels_b200 as tpk
from torch_points_kernels_b200.chamfer_dist import chamfer_dist
from torch_points_kernels_b200.gridding import gridding

DEV = "cuda"


def listed():
    return [
        # one small object classified as it comes in: every call is a few microseconds of GPU work,
        # so the latency of the calls themselves counts
        dict(name="infer_1x1024", kind="infer", shape="surface", batch=1, points=1024, levels=2, channels=32,
             nsample=32, radius=0.2, decoder=False),
        # one scan segmented as it comes in: the longest chain of dependent calls, with few blocks each
        dict(name="infer_1x16384", kind="infer", shape="surface", batch=1, points=16384, levels=4, channels=64,
             nsample=32, radius=0.1, decoder=True),
        # the training step that the benchmark is quoted on
        dict(name="train_16x16384", kind="train", shape="ball", batch=16, points=16384, levels=4, channels=64,
             nsample=32, radius=0.1, fused=False),
        # a training step at sizes that are multiples of nothing, with the fused grouping
        dict(name="train_3x10007", kind="train", shape="ball", batch=3, points=10007, levels=3, channels=35,
             nsample=24, radius=0.12, fused=True),
        # neighbour features between two resolutions of a small batch
        dict(name="search_4x4096", kind="search", batch=4, points=4096, queries=1024, channels=64, k=3,
             nsample=32, radius=0.2),
        # indoor scenes of very different sizes packed into one batch, as sparse networks take them
        dict(name="packed_64x110k", kind="packed", scenes=64, low=20000, high=200000, every=10, k=16,
             nsample=64, radius=0.05),
        # a few small crops in the same layout, every point its own query
        dict(name="packed_5x4k", kind="packed", scenes=5, low=501, high=8009, every=1, k=8, nsample=20,
             radius=0.25),
        # completion at full resolution: loss of a batch, both clouds trained
        dict(name="chamfer_32x16384", kind="chamfer", batch=32, points=16384, others=16384, both=True),
        # the coarse output of a completion network against its target
        dict(name="chamfer_64x2048", kind="chamfer", batch=64, points=2048, others=2048, both=False),
        # a batch of large scans thinned out, with the neighbourhoods of what is left
        dict(name="cloud_8x1048576", kind="cloud", batch=8, points=1048576, samples=65536, nsample=32,
             radius=0.02),
        # proposals of an instance segmentation and their overlap with the labels
        dict(name="segment_4x60k", kind="segment", scenes=4, points=60000, classes=8, nsample=16, radius=0.03),
        # the point/grid layers of a completion network
        dict(name="grnet_16x2048", kind="grnet", batch=16, points=2048, scale=32, channels=32),
    ]


def _spread(rng, low, high):
    """A whole number between the two, spread evenly over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _drawn(rng):
    kind = rng.choice(["infer", "train", "search", "packed", "chamfer", "cloud", "segment", "grnet"])
    if kind in ("infer", "train"):
        points = _spread(rng, 512, 32768)
        c = dict(kind=kind, shape=rng.choice(["ball", "surface"]), batch=_spread(rng, 1, 16 if kind == "train" else 8),
                 points=points, levels=rng.randint(1, 4 if points >= 4096 else 2), channels=_spread(rng, 16, 96),
                 nsample=rng.choice([16, 24, 32, 48, 64]),
                 radius=round(0.1 * (16384.0 / points) ** (1 / 3.0) * rng.uniform(0.8, 1.3), 3))
        if kind == "infer":
            c["decoder"] = rng.random() < 0.5
        else:
            c["fused"] = rng.random() < 0.5
        return c
    if kind == "search":
        points = _spread(rng, 256, 65536)
        return dict(kind=kind, batch=_spread(rng, 1, 8), points=points, queries=max(3, points // rng.choice([1, 2, 4, 8])),
                    channels=_spread(rng, 16, 128), k=rng.choice([1, 3, 8, 16, 24, 32]), nsample=rng.choice([16, 32, 64]),
                    radius=round((4096.0 / points) ** (1 / 3.0) * rng.uniform(0.1, 0.25), 4))
    if kind == "packed":
        low = _spread(rng, 500, 20000)
        return dict(kind=kind, scenes=_spread(rng, 1, 64), low=low, high=low * rng.randint(2, 10),
                    every=rng.choice([1, 2, 4, 10]), k=rng.choice([3, 8, 16, 20, 32]), nsample=rng.choice([16, 20, 32, 64]),
                    radius=round(0.05 * (20000.0 / low) ** 0.5 * rng.uniform(0.8, 1.3), 4))
    if kind == "chamfer":
        points = _spread(rng, 256, 16384)
        return dict(kind=kind, batch=_spread(rng, 1, 64), points=points,
                    others=points if rng.random() < 0.5 else _spread(rng, 256, 16384), both=rng.random() < 0.5)
    if kind == "cloud":
        points = _spread(rng, 65536, 1048576)
        return dict(kind=kind, batch=_spread(rng, 1, 8), points=points, samples=points // rng.choice([16, 24, 32, 64]),
                    nsample=rng.choice([16, 32, 64]), radius=round(0.02 * (1048576.0 / points) ** (1 / 3.0), 4))
    if kind == "segment":
        return dict(kind=kind, scenes=rng.randint(1, 4), points=_spread(rng, 5000, 60000), classes=rng.randint(2, 12),
                    nsample=rng.choice([12, 16, 24]), radius=0.03)
    return dict(kind=kind, batch=_spread(rng, 1, 16), points=_spread(rng, 512, 2048), scale=rng.choice([16, 24, 32]),
                channels=rng.choice([16, 24, 32]))


def draw(rng):
    """One more case of the same ranges that moves no more bytes than the largest listed case."""
    most = max(work(c)["bytes"] for c in listed())
    while True:
        c = _drawn(rng)
        if work(c)["bytes"] <= most:
            return c


# ---- inputs ----------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _objects(g, shape, batch, points):
    """(batch, points, 3): uniform in the unit ball, or on the surfaces of four ellipsoids in it."""
    d = _unit(_randn(g, batch, points, 3))
    if shape == "ball":
        return (d * _rand(g, batch, points, 1) ** (1.0 / 3.0)).contiguous()
    part = torch.randint(0, 4, (batch, points, 1), generator=g, device=DEV).expand(-1, -1, 3)
    centre = 0.5 * (2 * _rand(g, batch, 4, 3) - 1)
    axes = 0.1 + 0.35 * _rand(g, batch, 4, 3)
    return (d * axes.gather(1, part) + centre.gather(1, part)).contiguous()


def _level_sizes(case):
    """Points per level: what comes in, then a quarter of it per level."""
    return [case["points"] // 4 ** l for l in range(case["levels"] + 1)]


def _scene_sizes(case):
    """Sizes of the scenes of a packed batch: spread over the range, the same for every seed."""
    span = case["high"] - case["low"]
    return [case["low"] + int(span * ((0.5 + 0.6180339887 * s) % 1.0)) for s in range(case["scenes"])]


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("infer", "train"):
        sizes, b = _level_sizes(case), case["batch"]
        s = dict(case=case, xyz=_objects(g, case["shape"], b, case["points"]))
        s["sa"] = [_randn(g, b, case["channels"] << l, sizes[l]) for l in range(case["levels"])]
        s["fp"] = [_randn(g, b, case["channels"] << l, sizes[l + 1]) for l in range(case["levels"])]
        if kind == "train":
            rows = 3 if case["fused"] else 0
            s["g_grouped"] = [_randn(g, b, rows + (case["channels"] << l), sizes[l + 1], case["nsample"])
                              for l in range(case["levels"])]
            s["g_up"] = [_randn(g, b, case["channels"] << l, sizes[l]) for l in range(case["levels"])]
            for t in s["sa"] + s["fp"]:
                t.requires_grad_(True)
        return s
    if kind == "search":
        x = _rand(g, case["batch"], case["points"], 3)
        pick = _rand(g, case["batch"], case["points"]).argsort(dim=1)[:, :case["queries"], None].expand(-1, -1, 3)
        return dict(case=case, x=x, y=x.gather(1, pick).contiguous(),
                    features=_randn(g, case["batch"], case["channels"], case["queries"]))
    if kind == "packed":
        sizes = torch.tensor(_scene_sizes(case), device=DEV)
        scene = torch.repeat_interleave(torch.arange(len(sizes), device=DEV), sizes)
        n = scene.numel()
        plane = (_rand(g, n) * (3 + 5 * _rand(g, len(sizes)))[scene]).long()  # 3 to 8 planes of 5 m a scene
        axis = torch.randint(0, 3, (len(sizes), 8), generator=g, device=DEV)[scene, plane]
        x = 5.0 * _rand(g, n, 3)
        offset = 5.0 * _rand(g, len(sizes), 8)[scene, plane]
        x.scatter_(1, axis[:, None], offset[:, None])
        x = (x + 0.01 * _randn(g, n, 3)).contiguous()
        at = torch.arange(0, n, case["every"], device=DEV)
        return dict(case=case, x=x, batch_x=scene, y=x[at].contiguous(), batch_y=scene[at].contiguous())
    if kind == "chamfer":
        b, n, m = case["batch"], case["points"], case["others"]
        pred = _unit(_randn(g, b, n, 3))
        truth = _unit(_randn(g, b, m, 3))
        same = min(int(0.7 * m), n)  # most points of the other cloud lie near one of this cloud
        truth[:, :same] = pred[:, :same]
        truth = truth + 0.01 * _randn(g, b, m, 3)
        mix = _rand(g, b, m).argsort(dim=1)[:, :, None].expand(-1, -1, 3)
        return dict(case=case, pred=pred.contiguous().requires_grad_(True),
                    truth=truth.gather(1, mix).contiguous().requires_grad_(case["both"]))
    if kind == "cloud":
        b, n = case["batch"], case["points"]
        part = torch.randint(0, 32, (b, n, 1), generator=g, device=DEV).expand(-1, -1, 3)
        mean = _rand(g, b, 32, 3)
        sigma = torch.exp(_rand(g, b, 32, 3) * math.log(0.2 / 0.01) + math.log(0.01))
        return dict(case=case, xyz=(mean.gather(1, part) + _randn(g, b, n, 3) * sigma.gather(1, part)).contiguous())
    if kind == "segment":
        return _segment_scenes(case, g)
    b, n, c = case["batch"], case["points"], case["channels"]
    s = dict(case=case, points=(0.9 * (_rand(g, b, n, 3) - 0.5)).requires_grad_(True))
    s["maps"] = [_randn(g, b, c << l, 32 >> l, 32 >> l, 32 >> l).requires_grad_(True) for l in range(3)]
    s["g_grid"] = _randn(g, b, (2 * case["scale"]) ** 3)
    s["g_sampled"] = [_randn(g, b, n, 8, c << l) for l in range(3)]
    return s


def _segment_scenes(case, g):
    """Scenes of flat objects of about a thousand points, 2 cm between neighbours, over a background."""
    n, scenes = case["points"], case["scenes"]
    objects = max(2, n // 1000)
    total = n * scenes
    scene = torch.arange(scenes, device=DEV).repeat_interleave(n)
    instance = torch.randint(0, objects, (total,), generator=g, device=DEV)
    instance[_rand(g, total) < 0.3] = 0  # floor and walls: a third of the points, no instance
    centre = _rand(g, scenes, objects, 3) * torch.tensor([8.0, 8.0, 3.0], device=DEV)
    side = 0.02 * math.sqrt(0.7 * n / objects)
    axis = torch.randint(0, 3, (scenes, objects), generator=g, device=DEV)
    kind = 1 + torch.randint(0, case["classes"], (scenes, objects), generator=g, device=DEV)
    kind[:, 0] = 0
    d = _rand(g, total, 3) - 0.5
    d.scatter_(1, axis[scene, instance][:, None], 0.0)
    size = torch.where(instance == 0, 8.0, side)[:, None]
    pos = centre[scene, instance] + d * size + 0.002 * _randn(g, total, 3)
    return dict(case=case, pos=pos.contiguous(), labels=kind[scene, instance], batch=scene, instances=instance)


# ---- one pass --------------------------------------------------------------------------------


def _upsample(unknown, known, features):
    """Interpolation of a feature-propagation layer: weights inverse to the distance."""
    dist, idx = tpk.three_nn(unknown, known)
    w = 1.0 / (dist + 1e-8)
    return tpk.three_interpolate(features, idx, w / w.sum(dim=2, keepdim=True)), dist, idx


def _run_infer(s):
    c, out = s["case"], []
    xyz = [s["xyz"]]
    for l in range(c["levels"]):
        sampled = tpk.furthest_point_sample(xyz[l], xyz[l].shape[1] // 4)
        centres, idx, grouped = tpk.sa_group(xyz[l], s["sa"][l], sampled, c["radius"] * 2 ** l, c["nsample"])
        xyz.append(centres)
        out.append((sampled, centres, idx, grouped))
    if c["decoder"]:
        for l in reversed(range(c["levels"])):
            out.append(_upsample(xyz[l], xyz[l + 1], s["fp"][l]))
    return out


def _run_train(s):
    c, out = s["case"], []
    xyz, grouped, up = [s["xyz"]], [], []
    for l in range(c["levels"]):
        r = c["radius"] * 2 ** l
        if c["fused"]:
            sampled = tpk.furthest_point_sample(xyz[l], xyz[l].shape[1] // 4)
            centres, idx, rows = tpk.sa_group(xyz[l], s["sa"][l], sampled, r, c["nsample"])
            out.append((sampled, centres, idx))
        else:
            sampled, centres = tpk.furthest_point_sample(xyz[l], xyz[l].shape[1] // 4, return_xyz=True)
            idx, dist = tpk.ball_query(r, c["nsample"], xyz[l], centres, mode="dense")
            rows = tpk.grouping_operation(s["sa"][l], idx)
            out.append((sampled, centres, idx, dist))
        xyz.append(centres)
        grouped.append(rows)
    for l in reversed(range(c["levels"])):
        rows, dist, idx = _upsample(xyz[l], xyz[l + 1], s["fp"][l])
        up.insert(0, rows)
        out.append((dist, idx))
    grads = torch.autograd.grad(grouped + up, s["sa"] + s["fp"], s["g_grouped"] + s["g_up"])
    return out, [t.detach() for t in grouped + up], grads


def _run_grnet(s):
    c = s["case"]
    grid = gridding(s["points"], c["scale"])
    sampled = [tpk.cubic_feature_sampling(s["points"], m) for m in s["maps"]]
    grads = torch.autograd.grad([grid] + sampled, [s["points"]] + s["maps"], [s["g_grid"]] + s["g_sampled"])
    return grid.detach(), [t.detach() for t in sampled], grads


def _run_segment(s):
    """Per point the proposal that it belongs to (-1: none), and the overlaps of all proposals, in
    tables of fixed size: proposals have at least 32 points."""
    c, n = s["case"], s["pos"].shape[0]
    clusters = tpk.region_grow(s["pos"], s["labels"], s["batch"], ignore_labels=[0], nsample=c["nsample"],
                               radius=c["radius"])
    iou = tpk.instance_iou(clusters, s["instances"], s["batch"])
    proposal = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    sizes = torch.tensor([len(p) for p in clusters], device=DEV)
    proposal[torch.cat(clusters)] = torch.repeat_interleave(torch.arange(len(clusters), device=DEV), sizes)
    overlaps = torch.zeros((n // 32, iou.shape[1]), device=DEV)
    overlaps[:iou.shape[0]] = iou
    return proposal, overlaps


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "infer":
        return _run_infer(state)
    if kind == "train":
        return _run_train(state)
    if kind == "search":
        near = tpk.ball_query(c["radius"], c["nsample"], state["x"], state["y"], mode="dense")
        nearest = tpk.knn(state["x"], state["y"], c["k"])
        return near, nearest, _upsample(state["x"], state["y"], state["features"])
    if kind == "packed":
        near = tpk.ball_query(c["radius"], c["nsample"], state["x"], state["y"], mode="partial_dense",
                              batch_x=state["batch_x"], batch_y=state["batch_y"])
        return near, tpk.knn(state["x"], state["y"], c["k"], state["batch_x"], state["batch_y"])
    if kind == "chamfer":
        loss = chamfer_dist(state["pred"], state["truth"])
        trained = [state["pred"], state["truth"]] if c["both"] else [state["pred"]]
        return loss.detach(), torch.autograd.grad(loss, trained)
    if kind == "cloud":
        sampled, centres = tpk.furthest_point_sample(state["xyz"], c["samples"], return_xyz=True)
        return sampled, centres, tpk.ball_query(c["radius"], c["nsample"], state["xyz"], centres, mode="dense")
    if kind == "segment":
        return _run_segment(state)
    return _run_grnet(state)


# ---- what a pass cannot do without -------------------------------------------------------------
# Bytes: every call reads its inputs once and writes its results once.  Operations: one squared
# distance (8) for each neighbour that is returned and for each point that is sampled from, one
# multiply-add (2) for each value that is weighted or summed.


def _sampling(b, n, m, coords):
    return 12 * b * n + (16 if coords else 4) * b * m, 8 * b * n


def _ball(b, n, m, k):
    return 12 * b * (n + m) + 12 * b * m * k, 8 * b * m * k


def _three(b, n, m):
    return 12 * b * (n + m) + 24 * b * n, 24 * b * n


def _interpolate(b, c, n, m):
    return 4 * b * c * (n + m) + 24 * b * n, 6 * b * c * n


def work(case):
    kind, parts = case["kind"], []
    if kind in ("infer", "train"):
        sizes, b, ns = _level_sizes(case), case["batch"], case["nsample"]
        fused = kind == "infer" or case["fused"]
        for l in range(case["levels"]):
            n, m, c = sizes[l], sizes[l + 1], case["channels"] << l
            parts.append(_sampling(b, n, m, not fused))
            rows = 4 * b * c * (n + m * ns)
            if fused:
                parts.append((12 * b * (n + 2 * m) + 8 * b * m * ns + rows + 12 * b * m * ns, 8 * b * m * ns))
            else:
                parts.append(_ball(b, n, m, ns))
                parts.append((8 * b * m * ns + rows, 0))
            if kind == "train" or case["decoder"]:
                parts += [_three(b, n, m), _interpolate(b, c, n, m)]
            if kind == "train":
                parts += [(8 * b * m * ns + rows, b * c * m * ns), _interpolate(b, c, n, m)]
    elif kind == "search":
        b, n, m = case["batch"], case["points"], case["queries"]
        parts += [_ball(b, n, m, case["nsample"]), _ball(b, n, m, case["k"]), _three(b, n, m),
                  _interpolate(b, case["channels"], n, m)]
    elif kind == "packed":
        n = sum(_scene_sizes(case))
        m = -(-n // case["every"])
        parts += [(20 * (n + m) + 12 * m * k, 8 * m * k) for k in (case["nsample"], case["k"])]
    elif kind == "chamfer":
        b, n, m = case["batch"], case["points"], case["others"]
        parts += [(12 * b * (n + m), 8 * b * (n + m)), (12 * b * (n + m) + 12 * b * (n + (m if case["both"] else 0)), 6 * b * (n + m))]
    elif kind == "cloud":
        b, n, m = case["batch"], case["points"], case["samples"]
        parts += [_sampling(b, n, m, True), _ball(b, n, m, case["nsample"])]
    elif kind == "segment":
        n = case["scenes"] * case["points"]
        parts.append((36 * n + 8 * n, 8 * n * case["nsample"]))
    else:
        b, n = case["batch"], case["points"]
        cells = (2 * case["scale"]) ** 3
        parts.append((2 * 12 * b * n + 2 * 4 * b * cells, 2 * 48 * b * n))
        for l in range(3):
            c = case["channels"] << l
            parts.append((2 * 4 * b * c * (32 >> l) ** 3 + 2 * 4 * b * n * 8 * c + 2 * 12 * b * n, 8 * b * n * c))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    """Indices are the same; coordinates and squared distances are too, up to the last bits of their
    32-bit arithmetic; interpolated values and gradients are 32-bit sums of some tens of terms in any order."""
    if case["kind"] == "packed":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 1e-5, "max": 1e-3}
