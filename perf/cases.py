"""Measured cases of the evaluators: what each passes through the public API, over the sizes it is used at.

A case names a path (``kind``), its sizes and its options. ``prepare`` makes seeded inputs on the GPU (stuff regions
around random sites, things as random ellipses, predictions and detections as perturbed copies of the target),
``run`` makes one pass and ``exact`` restates its results in 64 bits with plain torch and numpy.

The reward server is not a case of its own: its batches are the reward and prefix passes below behind a request queue,
and what it is judged by (latency under an arrival schedule) is not the time of a pass.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import panoptic_evaluator_gb300 as pe
from panoptic_evaluator_gb300.ragged import SegmentationImages

DEVICE = "cuda"
PREFIX_IOU = (0.5, 0.75)


def listed():
    return [
        # One generated segmentation scored while a policy is trained or served: latency and launches count.
        dict(name="reward_one", kind="reward", images=1, height=480, width=640, slots=41, classes=133, validate=True),
        # A group of rollouts scored together.
        dict(name="reward_group", kind="reward", images=16, height=512, width=512, slots=64, classes=133,
             validate=False),
        # A small evaluation batch of few segments and classes.
        dict(name="panoptic_small", kind="panoptic", images=8, height=256, width=256, slots=32, classes=20,
             validate=True),
        # A validation batch of COCO images on a padded canvas, slot capacity above the segments in use.
        dict(name="panoptic_coco", kind="panoptic", images=16, height=640, width=640, spread=160, slots=101,
             classes=133, validate=False),
        # Decoded COCO panoptic PNGs (RGB identifiers) and their segments_info, straight from the files.
        dict(name="panoptic_png", kind="png", images=8, height=427, width=640, slots=41, classes=133, validate=True),
        # The usual evaluation loop of one image per update, odd height: rows at any byte offset.
        dict(name="instance_one", kind="instance", images=1, height=427, width=640, spread=0, dets=100, targets=20,
             classes=80, validate=True),
        # A batch of COCO images of their own sizes, 100 detections each.
        dict(name="instance_coco", kind="instance", images=32, height=640, width=640, spread=160, dets=100,
             targets=50, classes=80, validate=False),
        # The same detections on one padded canvas, as a model's postprocessor leaves them.
        dict(name="instance_canvas", kind="instance", images=16, height=640, width=640, spread=0, dets=100,
             targets=50, classes=80, validate=False),
        # Joint PQ and AP of a fixed-size batch with many segments and detections per image, few classes.
        dict(name="combined_batch", kind="combined", images=8, height=512, width=768, slots=257, dets=256,
             classes=15, validate=False),
        # Joint PQ and AP over uneven images packed once and evaluated in one call: dataset throughput.
        dict(name="combined_images", kind="arena", images=64, height=1024, width=1024, spread=704, slots=150,
             dets=100, classes=133, validate=False),
        # One generated sequence of masks, the score after every eighth mask.
        dict(name="prefix_one", kind="prefix", images=1, height=256, width=384, slots=101, masks=64, every=8,
             classes=133, validate=True),
        # A group of generated sequences of one image size, odd sides, scored half way and at the end.
        dict(name="prefix_group", kind="prefix", images=16, height=845, width=845, slots=101, masks=64, every=32,
             classes=133, validate=False),
    ]


def _between(rng, low, high):
    """A whole number, its logarithm spread evenly."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))))))


def draw(rng):
    kind = rng.choice(("reward", "panoptic", "png", "instance", "instance", "combined", "arena", "prefix"))
    case = dict(kind=kind, classes=rng.choice((15, 20, 80, 133)), validate=rng.random() < 0.4)
    if kind in ("reward", "panoptic", "png"):
        case.update(images=_between(rng, 1, 16), height=_between(rng, 97, 768), width=_between(rng, 97, 768),
                    slots=_between(rng, 10, 150))
        if kind == "png":
            case["images"] = min(case["images"], 8)
        if kind == "panoptic":
            case["spread"] = rng.choice((0, min(case["height"], case["width"]) // 4))
    elif kind == "instance":
        case.update(images=_between(rng, 1, 32), height=rng.randint(320, 640), width=rng.randint(320, 640),
                    spread=rng.choice((0, 0, 97, 160)), dets=_between(rng, 10, 120), targets=_between(rng, 2, 80),
                    classes=rng.choice((1, 20, 80)))
    elif kind == "combined":
        case.update(images=_between(rng, 1, 8), height=_between(rng, 256, 640), width=_between(rng, 256, 768),
                    slots=_between(rng, 10, 257), dets=_between(rng, 5, 256))
    elif kind == "arena":
        case.update(images=_between(rng, 4, 48), height=1024, width=1024, spread=rng.choice((384, 704)),
                    slots=_between(rng, 20, 150), dets=_between(rng, 10, 100))
    else:
        case.update(images=_between(rng, 1, 16), height=_between(rng, 128, 845), width=_between(rng, 128, 845),
                    slots=_between(rng, 10, 150), masks=_between(rng, 16, 64), every=rng.choice((8, 16, 32)))
        case["every"] = max(case["every"], -(-case["masks"] * case["images"] // 32))  # at most 32 snapshots are read
    return case


# ---- inputs --------------------------------------------------------------------------------------------------------


class _Random:
    """Seeded draws on the GPU and, for sizes and tables, on the host."""

    def __init__(self, seed):
        self.host = np.random.default_rng(seed)
        self.device = torch.Generator(DEVICE).manual_seed(int(self.host.integers(1 << 62)))

    def uniform(self, shape, low=0.0, high=1.0):
        return torch.rand(shape, device=DEVICE, generator=self.device) * (high - low) + low

    def below(self, shape, high):
        return torch.randint(0, high, shape, device=DEVICE, generator=self.device)


def _things(classes):
    return max(1, classes * 3 // 5)


def _ellipses(r, n, h, w, largest=20000.0):
    """Parameters [n, 5] (centre y, x, two half axes, angle) of ellipses, areas log-uniform from 32 pixels."""
    area = torch.exp(r.uniform(n, math.log(32.0), math.log(largest)))
    ratio = r.uniform(n, 0.5, 2.0)
    return torch.stack((r.uniform(n, 0, h - 1), r.uniform(n, 0, w - 1), (area / math.pi * ratio).sqrt(),
                        (area / math.pi / ratio).sqrt(), r.uniform(n, 0, math.pi)), 1)


def _perturbed(r, shapes, h, w):
    """Shapes shifted by up to 8 pixels and grown or shrunk by up to 5."""
    out = shapes.clone()
    out[:, :2] += r.uniform((len(shapes), 2), -8, 8)
    out[:, 0].clamp_(0, h - 1)
    out[:, 1].clamp_(0, w - 1)
    out[:, 2:4] = (out[:, 2:4] + r.uniform((len(shapes), 1), -5, 5)).clamp_min(2.0)
    return out


def _masks(shapes, h, w):
    """Bool [n, h, w] masks of the ellipses; the centre pixel always belongs to its mask."""
    out = torch.empty((len(shapes), h, w), dtype=torch.bool, device=DEVICE)
    y = torch.arange(h, device=DEVICE, dtype=torch.float32)[None, :, None]
    x = torch.arange(w, device=DEVICE, dtype=torch.float32)[None, None, :]
    for at in range(0, len(shapes), 32):
        cy, cx, a, b, t = (v[:, None, None] for v in shapes[at:at + 32].unbind(1))
        dy, dx, c, s = y - cy, x - cx, torch.cos(t), torch.sin(t)
        out[at:at + 32] = ((dx * c + dy * s) / a) ** 2 + ((dy * c - dx * s) / b) ** 2 <= 1
    row = torch.arange(len(shapes), device=DEVICE)
    out[row, shapes[:, 0].round().long(), shapes[:, 1].round().long()] = True
    return out


def _counts(labels, n):
    return torch.bincount(labels.reshape(-1).long(), minlength=n)[:n]


def _scene(r, h, w, slots, classes, void=0.03):
    """A target: stuff regions around random sites, things drawn over them, some void.

    Returns the map, its class table, crowd flags and the things' shapes with their slots.
    """
    things, stuff = _things(classes), min(8, max(1, (slots - 1) // 3))
    y = torch.arange(h, device=DEVICE, dtype=torch.float32)[:, None]
    x = torch.arange(w, device=DEVICE, dtype=torch.float32)[None]
    sites = r.uniform((stuff, 2)) * torch.tensor([h, w], device=DEVICE)
    target = torch.stack([(y - s[0]) ** 2 + (x - s[1]) ** 2 for s in sites]).argmin(0).int() + 1
    n = slots - 1 - stuff
    shapes = _ellipses(r, n, h, w)
    slot = torch.arange(n, device=DEVICE, dtype=torch.int32) + stuff + 1
    for at in range(0, n, 32):  # later things cover earlier ones
        covered = _masks(shapes[at:at + 32], h, w) * slot[at:at + 32, None, None]
        target = torch.maximum(target, covered.amax(0))
    target[r.uniform((h, w)) < void] = 0
    table = torch.cat((things + r.below((stuff,), max(1, classes - things)), r.below((n,), things))).int()
    table = torch.cat((torch.full((1,), -1, device=DEVICE, dtype=torch.int32), table.clamp_max(classes - 1)))
    table[_counts(target, slots) == 0] = -1
    crowd = (r.uniform(slots) < 0.02) & (table >= 0) & (table < things)
    return target, table, crowd, shapes, slot


def _prediction(r, target, table, classes, capacity):
    """The target with a tenth of its pixels relabelled from a neighbour, segments split and merged, classes flipped."""
    h, w = target.shape
    slots = len(table)
    which = r.below((h, w), 40)
    pred = target.clone()
    for k, (dy, dx) in enumerate(((1, 0), (-1, 0), (0, 1), (0, -1))):
        pred = torch.where(which == k, target.roll((dy, dx), (0, 1)), pred)
    ids = torch.arange(slots, device=DEVICE)
    merged = torch.where(r.uniform(slots) < 0.03, r.below((slots,), slots).clamp_min(1), ids)
    merged[0] = 0
    split = (r.uniform(slots) < 0.05) & (ids > 0)
    room = capacity - slots
    extra = torch.cumsum(split, 0)
    split &= extra <= room
    right = torch.where(split, slots - 1 + extra, merged)
    side = torch.arange(w, device=DEVICE)[None] > (r.uniform(()) * w)
    pred = torch.where(side, right[pred.long()], merged[pred.long()]).int()
    out = torch.full((capacity,), -1, device=DEVICE, dtype=torch.int32)
    out[:slots] = table
    out[right[split]] = table[split]
    labels = r.below((capacity,), classes).int()
    out = torch.where((out < 0) | (r.uniform(capacity) < 0.1), labels, out)
    out[_counts(pred, capacity) == 0] = -1
    out[0] = -1
    return pred, out


def _detections(r, shapes, labels, n, h, w, classes, share):
    """n masks: `share` of them perturbed copies of the shapes, the others anywhere; their classes and scores."""
    copies = int(round(n * share)) if len(shapes) else 0
    pick = r.below((copies,), max(1, len(shapes)))
    parts = ([_perturbed(r, shapes[pick], h, w)] if copies else []) + [_ellipses(r, n - copies, h, w)]
    found = r.below((n,), classes)
    found[:copies] = torch.where(r.uniform(copies) < 0.9, labels[pick].long(), found[:copies])
    scores = np.concatenate((r.host.beta(5, 2, copies), r.host.beta(2, 5, n - copies))).astype(np.float32)
    mix = torch.from_numpy(r.host.permutation(n)).to(DEVICE)
    return _masks(torch.cat(parts)[mix], h, w), found[mix], torch.from_numpy(scores).to(DEVICE)[mix]


def _side(r, case, key):
    return case[key] - int(r.host.integers(0, case.get("spread", 0) + 1))


def _padded(image, case, slots):
    """The image on the batch's canvas (void outside it), its tables at the batch's slot capacity."""
    h, w = image["target"].shape
    for key in ("target", "pred"):
        if key in image:
            image[key] = torch.nn.functional.pad(image[key], (0, case["width"] - w, 0, case["height"] - h))
    for key, size, fill in (("gc", slots, -1), ("crowd", slots, False), ("pc", slots + 20, -1)):
        if key in image:
            image[key] = torch.nn.functional.pad(image[key], (0, size - len(image[key])), value=fill)
    return image


def _images(case, seed):
    """One dict of plain tensors for each image of the case."""
    r, out = _Random(seed), []
    classes, kind = case["classes"], case["kind"]
    for _ in range(case["images"]):
        h, w = _side(r, case, "height"), _side(r, case, "width")
        if kind == "instance":
            n = case["targets"] if case["images"] == 1 else int(r.host.integers(1, case["targets"] + 1))
            shapes, labels = _ellipses(r, n, h, w), r.below((n,), classes)
            masks, found, scores = _detections(r, shapes, labels, case["dets"], h, w, classes, 0.7)
            out.append(dict(masks=masks, det_classes=found, scores=scores, gt_masks=_masks(shapes, h, w),
                            gt_classes=labels, crowd=r.uniform(n) < 0.02))
            continue
        # Images have their own segment counts; a batch's tables have room for the largest.
        slots, dets = case["slots"], case.get("dets", 0)
        if case["images"] > 1 and kind != "combined":
            slots = int(r.host.integers(10, slots + 1))
        if kind == "arena":
            dets = int(r.host.integers(5, dets + 1))
        target, table, crowd, shapes, slot = _scene(r, h, w, slots, classes)
        image = dict(target=target, gc=table, crowd=crowd)
        if kind == "prefix":
            things = (table[slot.long()] >= 0).nonzero()[:, 0]
            image["masks"], found, _ = _detections(r, shapes[things], table[slot[things].long()], case["masks"], h, w,
                                                   classes, 0.8)
            image["det_classes"] = found.int()
        else:
            image["pred"], image["pc"] = _prediction(r, target, table, classes, slots + 20)
        if dets:
            things = (table[slot.long()] >= 0).nonzero()[:, 0]
            image["masks"], image["det_classes"], image["scores"] = _detections(
                r, shapes[things], table[slot[things].long()], dets, h, w, _things(classes), 0.85)
        out.append(image if kind == "arena" else _padded(image, case, case["slots"]))
    return out


def _stack(images, key):
    return torch.stack([i[key] for i in images])


def _png(r, maps, tables, crowds):
    """RGB identifiers [B, H, W, 3] and segments_info of slot maps."""
    rgb, info = [], []
    for labels, table, crowd in zip(maps, tables, crowds):
        ids = np.concatenate(([0], 1 + r.host.choice((1 << 24) - 1, len(table) - 1, replace=False)))
        palette = torch.from_numpy(np.stack((ids % 256, ids // 256 % 256, ids // 65536), 1).astype(np.uint8))
        rgb.append(palette.to(DEVICE)[labels.long()])
        info.append([dict(id=int(ids[s]), category_id=int(c), iscrowd=int(k))
                     for s, (c, k) in enumerate(zip(table.tolist(), crowd.tolist())) if c >= 0])
    return torch.stack(rgb), info


def prepare(case, seed):
    images, kind, classes = _images(case, seed), case["kind"], case["classes"]
    isthing = [c < _things(classes) for c in range(classes)]
    state = dict(case=case, isthing=isthing)
    if kind == "instance":
        keys = ("masks", "det_classes", "scores")
        state["prediction"] = pe.InstanceBatch(*[[i[k] for i in images] for k in keys])
        state["target"] = pe.InstanceBatch([i["gt_masks"] for i in images], [i["gt_classes"] for i in images],
                                           crowd=[i["crowd"] for i in images])
        state["evaluator"] = pe.InstanceEvaluator(classes, validate=case["validate"])
        return state
    if kind == "arena":
        fields = ("target", "gc", "crowd", "pred", "pc", "masks", "det_classes", "scores")
        state["images"] = SegmentationImages(*[[i[f].cpu().numpy() for i in images] for f in fields], device=DEVICE)
        state["evaluator"] = pe.SegmentationEvaluator(classes, isthing=isthing, validate=case["validate"])
        return state
    if kind == "png":
        r = _Random(seed + 1)
        none = [torch.zeros(len(i["pc"]), dtype=torch.bool) for i in images]
        state["target"] = _png(r, [i["target"] for i in images], [i["gc"] for i in images],
                               [i["crowd"] for i in images])
        state["prediction"] = _png(r, [i["pred"] for i in images], [i["pc"] for i in images], none)
        state["evaluator"] = pe.PanopticEvaluator(classes, isthing=isthing, validate=case["validate"])
        return state
    state["target"] = pe.PanopticBatch(_stack(images, "target"), _stack(images, "gc"), _stack(images, "crowd"))
    if kind == "prefix":
        state["prediction"] = pe.InstanceBatch([i["masks"] for i in images], [i["det_classes"] for i in images])
        state["checkpoints"] = _checkpoints(case)
        return state
    state["prediction"] = pe.PanopticBatch(_stack(images, "pred"), _stack(images, "pc"))
    if kind == "panoptic":
        state["evaluator"] = pe.PanopticEvaluator(classes, isthing=isthing, validate=case["validate"])
    if kind == "combined":
        state["detections"] = pe.InstanceBatch(*[[i[k] for i in images] for k in ("masks", "det_classes", "scores")])
        state["evaluator"] = pe.SegmentationEvaluator(classes, isthing=isthing, validate=case["validate"])
    return state


def _checkpoints(case):
    points = list(range(case["every"], case["masks"] + 1, case["every"]))
    return points if points and points[-1] == case["masks"] else points + [case["masks"]]


def run(state):
    case = state["case"]
    kind, classes = case["kind"], case["classes"]
    if kind == "reward":
        return pe.panoptic_quality(state["prediction"], state["target"], classes, validate=case["validate"])
    if kind == "prefix":
        return _read_prefixes(case, pe.segmentation_prefixes(
            state["prediction"], state["target"], classes, isthing=state["isthing"],
            checkpoints=state["checkpoints"], iou_thresholds=PREFIX_IOU, validate=case["validate"]))
    evaluator = state["evaluator"]
    evaluator.reset()
    if kind == "png":
        categories = range(classes)
        (rgb, info), (pred_rgb, pred_info) = state["target"], state["prediction"]
        target = pe.PanopticBatch.from_coco(rgb, info, categories)
        evaluator.update(pe.PanopticBatch.from_coco(pred_rgb, pred_info, categories), target)
    elif kind == "arena":
        evaluator.update_images(state["images"])
    elif kind == "combined":
        evaluator.update(state["prediction"], state["detections"], state["target"])
    else:
        evaluator.update(state["prediction"], state["target"])
    return evaluator.compute()


def _read_prefixes(case, sequences):
    """What is read of each snapshot: everything counted for one sequence, the canvas scores for a group."""
    if case["images"] == 1 and len(sequences[0]) <= 8:
        return [dict(confusion=s["confusion"], iou_sum=s["iou_sum"], fp=s["fp"], miou=s["miou"],
                     tp=s["instance"]["tp"], precision=s["instance"]["precision"], recall=s["instance"]["recall"])
                for s in sequences[0]]
    return [[dict(confusion=s["confusion"], iou_sum=s["iou_sum"]) for s in q] for q in sequences]


def work(case):
    """Bytes of the maps and masks, each read once, and of the results; counting takes no floating-point work."""
    kind, classes = case["kind"], case["classes"]
    smaller = case["spread"] / 2 if kind in ("instance", "arena") else 0
    size = case["images"] * (case["height"] - smaller) * (case["width"] - smaller)
    scores = 8 * (classes * (classes + 9))
    curves = 8 * (10 * 102 * classes * 12)
    if kind == "reward":
        return dict(bytes=8 * size + 8 * case["images"], flops=0)
    if kind == "png":
        return dict(bytes=6 * size + scores, flops=0)
    if kind == "panoptic":
        return dict(bytes=8 * size + scores, flops=0)
    if kind == "instance":
        targets = case["targets"] if case["images"] == 1 else (case["targets"] + 1) / 2
        return dict(bytes=size * (case["dets"] + targets) + curves, flops=2 * size * case["dets"] * targets)
    if kind == "prefix":
        rows = case["images"] * len(_checkpoints(case))
        return dict(bytes=size * (4 + case["masks"]) + rows * scores, flops=0)
    dets = case["dets"] if kind == "combined" else (case["dets"] + 5) / 2
    return dict(bytes=size * (8 + dets) + scores + curves, flops=0)


# ---- results in 64 bits ----------------------------------------------------------------------------------------------


def _pairs(a, b, n, m):
    return torch.bincount((a.reshape(-1).long() * m + b.reshape(-1).long()), minlength=n * m).reshape(n, m).cpu().numpy()


def _match_panoptic(pairs, gc, pc, crowd, classes, reward=False):
    """tp, fp, fn [C], IoU sums [C] and confusion [C, C + 1] of one image's target x prediction pixel counts."""
    ga, pa = pairs.sum(1), pairs.sum(0)
    iou = pairs / np.maximum(ga[:, None] + pa[None] - pairs - pairs[:1], 1)
    same = (gc[:, None] == pc[None]) & (gc >= 0)[:, None]
    match = same & ~crowd[:, None] & (iou > 0.5)
    ignored = pairs[0].copy()
    for g in np.flatnonzero(crowd):
        ignored = np.where(same[g], pairs[0] + pairs[g], ignored)  # the last crowd segment of the class
    wrong = (pc >= 0) & ~match.any(0) & (2 * ignored <= pa)
    if reward:
        wrong &= pa > 0
    missed = (gc >= 0) & ~crowd & ~match.any(1)
    count = lambda labels: np.bincount(labels, minlength=classes)  # noqa: E731
    tp, fp, fn = count(pc[match.any(0)]), count(pc[wrong]), count(gc[missed])
    sums = np.bincount(pc[match.any(0)], weights=(iou * match).sum(0)[match.any(0)], minlength=classes)
    confusion = np.zeros((classes, classes + 1), np.int64)
    rows = np.flatnonzero((gc >= 0) & ~crowd)
    np.add.at(confusion, (gc[rows][:, None], np.where(pc >= 0, pc, classes)[None]), pairs[rows])
    return tp, fp, fn, sums, confusion


def _panoptic_result(parts, classes):
    tp, fp, fn, sums, confusion = (sum(p[k] for p in parts) for k in range(5))
    thing = np.arange(classes) < _things(classes)
    weight = tp + 0.5 * (fp + fn)
    values = dict(pq=sums / np.maximum(weight, 1), sq=sums / np.maximum(tp, 1), rq=tp / np.maximum(weight, 1))
    result = {}
    for name, mask in (("All", thing | True), ("Things", thing), ("Stuff", ~thing)):
        mask = mask & (weight > 0)
        result[name] = {k: v[mask].sum() / max(1, mask.sum()) for k, v in values.items()}
        result[name]["n"] = int(mask.sum())
    hit = np.diagonal(confusion).astype(np.float64)
    union = confusion.sum(1) + confusion[:, :classes].sum(0) - hit
    values["iou"] = np.where(union > 0, hit / np.maximum(union, 1), np.nan)
    result.update(per_class=values, miou=np.nansum(values["iou"]) / max(1, (union > 0).sum()), tp=tp, fp=fp, fn=fn,
                  iou_sum=sums, confusion=confusion)
    return result


def _host(image, *keys):
    return [image[k].cpu().numpy() for k in keys]


def _panoptic_part(image, classes, reward=False):
    pairs = _pairs(image["target"], image["pred"], len(image["gc"]), len(image["pc"]))
    gc, pc, crowd = _host(image, "gc", "pc", "crowd")
    return _match_panoptic(pairs, gc, pc, crowd, classes, reward)


_AREAS = ((0, 1e10), (0, 32.0 ** 2), (32.0 ** 2, 96.0 ** 2), (96.0 ** 2, 1e10))


def _match_instances(inter, pa, ga, labels, targets, crowd, classes, records, positives):
    """Greedy matching of one image, detections by falling score: adds [40] outcomes of each to `records`."""
    iou = inter / np.maximum(np.where(crowd[None], pa[:, None], pa[:, None] + ga[None] - inter), 1)
    threshold = np.tile(np.linspace(0.5, 0.95, 10), 4)
    low, high = np.repeat(np.array(_AREAS), 10, 0).T
    outside = (ga[None] < low[:, None]) | (ga[None] > high[:, None]) | crowd[None]  # [40, G]
    np.add.at(positives, targets[targets >= 0], ~outside.reshape(4, 10, -1)[:, 0].T[targets >= 0])
    used, seen = np.zeros(outside.shape, bool), np.zeros(classes, np.int64)
    for d, c in enumerate(labels):
        seen[c] += 1
        state = np.where((pa[d] < low) | (pa[d] > high), -1, 0)
        of = np.flatnonzero(targets == c)
        if seen[c] <= 100 and len(of):
            free = (~used[:, of] | crowd[of]) & (iou[d, of] >= threshold[:, None])
            # In-range targets before ignored ones, then the largest IoU, the later target on equal ones.
            rank = np.where(free, iou[d, of] + 2 * ~outside[:, of], -1)[:, ::-1]
            best = len(of) - 1 - rank.argmax(1)
            taken = np.flatnonzero(rank.max(1) >= 0)
            used[taken, of[best[taken]]] = True
            state[taken] = np.where(outside[taken, of[best[taken]]], -1, 1)
        records.append((c, seen[c], state))


def _instance_result(records, scores, positives, classes):
    order = np.argsort(-scores, kind="stable")
    labels = np.array([r[0] for r in records])[order]
    ranks = np.array([r[1] for r in records])[order]
    states = np.stack([r[2] for r in records])[order]
    precision, recall = np.full((10, 101, classes, 4, 3), -1.0), np.full((10, classes, 4, 3), -1.0)
    for c in range(classes):
        rows = np.flatnonzero(labels == c)
        for m, most in enumerate((1, 10, 100)):
            chosen = states[rows[ranks[rows] <= most]].T.reshape(4, 10, -1)
            for a in np.flatnonzero(positives[c]):
                precision[:, :, c, a, m] = recall[:, c, a, m] = 0
                if not chosen.shape[2]:
                    continue
                tp, fp = (chosen[a] == 1).cumsum(1), (chosen[a] == 0).cumsum(1)
                reached, rate = tp / positives[c, a], tp / (tp + fp + np.finfo(np.float64).eps)
                rate = np.maximum.accumulate(rate[:, ::-1], 1)[:, ::-1]
                for t in range(10):
                    at = np.searchsorted(reached[t], np.arange(101) * 0.01, side="left")
                    precision[t, :, c, a, m] = np.append(rate[t], 0)[at]
                recall[:, c, a, m] = reached[:, -1]

    def mean(v):
        return v[v >= 0].mean() if (v >= 0).any() else -1.0

    result = dict(ap=mean(precision[:, :, :, 0, 2]), ap50=mean(precision[0, :, :, 0, 2]),
                  ap75=mean(precision[5, :, :, 0, 2]), precision=precision, recall=recall)
    for a, name in enumerate(("small", "medium", "large"), 1):
        result["ap_" + name], result["ar_" + name] = mean(precision[:, :, :, a, 2]), mean(recall[:, :, a, 2])
    for m, most in enumerate((1, 10, 100)):
        result["ar%d" % most] = mean(recall[:, :, 0, m])
    return result


def _instances(images, classes, shared):
    """AP results; `shared`: the targets are the thing segments of the panoptic map, else masks of their own."""
    records, scores, positives = [], [], np.zeros((classes, 4), np.int64)
    for i in images:
        order = torch.argsort(-i["scores"].double(), stable=True)
        masks = i["masks"][order]
        labels = i["det_classes"][order].cpu().numpy()
        if shared:
            n = len(i["gc"])
            inter = np.stack([_counts(i["target"][m], n).cpu().numpy() for m in masks])
            targets, ga = i["gc"].cpu().numpy(), _counts(i["target"], n).cpu().numpy()
            targets = np.where(targets < _things(classes), targets, -1)
        else:
            flat = i["gt_masks"].flatten(1)
            inter = np.stack([(flat & m.reshape(1, -1)).sum(1).cpu().numpy() for m in masks])
            targets, ga = i["gt_classes"].cpu().numpy(), flat.sum(1).cpu().numpy()
        pa = masks.flatten(1).sum(1).cpu().numpy()
        _match_instances(inter.astype(np.float64), pa, ga, labels, targets, i["crowd"].cpu().numpy(), classes,
                         records, positives)
        scores.append(i["scores"][order].double().cpu().numpy())
    return _instance_result(records, np.concatenate(scores), positives, classes)


def _prefix_result(image, case):
    classes, points = case["classes"], _checkpoints(case)
    gc, crowd, labels = _host(image, "gc", "crowd", "det_classes")
    masks, target, n = image["masks"], image["target"], len(gc)
    ga = _counts(target, n).cpu().numpy()
    canvas = torch.zeros(target.shape, dtype=torch.int64, device=DEVICE)
    tp, fp = np.zeros((2, classes), np.int64), np.zeros((2, classes), np.int64)
    positives = np.bincount(gc[(gc >= 0) & (gc < _things(classes)) & ~crowd], minlength=classes)
    used, out = np.zeros((2, n), bool), []
    for k, c in enumerate(labels):
        inter = _counts(target[masks[k]], n).cpu().numpy()
        canvas[masks[k]] = k + 1
        if c < _things(classes):
            area = inter.sum()
            iou = inter / np.maximum(np.where(crowd, area, area + ga - inter), 1)
            for t, threshold in enumerate(PREFIX_IOU):
                reached = (gc == c) & (iou >= threshold)
                free = reached & ~crowd & ~used[t]
                if free.any():
                    used[t, np.where(free, iou, -1).argmax()] = True
                    tp[t, c] += 1
                elif not (reached & crowd).any():
                    fp[t, c] += 1
        if k + 1 in points:
            pairs = _pairs(target, canvas, n, len(labels) + 1)
            pc = np.where(pairs.sum(0) > 0, np.concatenate(([-1], labels)), -1)
            r = _panoptic_result([_match_panoptic(pairs, gc, pc, crowd, classes)], classes)
            r["instance"] = dict(tp=tp.copy(), precision=tp / np.maximum(tp + fp, 1),
                                 recall=tp / np.maximum(positives, 1))
            out.append(r)
    return out


def exact(case, seed):
    images, kind, classes = _images(case, seed), case["kind"], case["classes"]
    if kind == "prefix":
        return _read_prefixes(case, [_prefix_result(i, case) for i in images])
    if kind == "instance":
        return _instances(images, classes, False)
    if kind == "reward":
        out = []
        for i in images:
            tp, fp, fn, sums, _ = _panoptic_part(i, classes, True)
            weight = tp + 0.5 * (fp + fn)
            out.append((sums / np.maximum(weight, 1)).sum() / max(1, (weight > 0).sum()))
        return np.array(out)
    result = _panoptic_result([_panoptic_part(i, classes) for i in images], classes)
    if kind in ("combined", "arena"):
        result["instance"] = _instances(images, classes, True)
    return result
