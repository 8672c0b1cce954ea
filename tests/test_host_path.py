"""The C++ host path against the Python path it stands in for.

On the CPU: both fill the same descriptor, offset, contraction and step tables. On the GPU: every
call gives the same results, errors and state through both, whatever form its arguments take.
"""

import contextlib
import ctypes
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from panoptic_evaluator_gb300 import InstanceBatch, PanopticBatch
from panoptic_evaluator_gb300 import _native as N

CTAS = 152


@pytest.fixture
def host():
    from panoptic_evaluator_gb300 import build
    build.build()
    return N.host()


@pytest.fixture
def on_cpu(monkeypatch):
    """The Python path's tables on CPU tensors: no pinned memory, no device queries."""
    empty = torch.empty
    monkeypatch.setattr(N, "sm_count", lambda device: CTAS)
    monkeypatch.setattr(N, "stream_handle", lambda device=None: 0)
    monkeypatch.setattr(N, "on_device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **k: empty(*a, **k))


def _instances(rng, B, aligned, dtypes=None, crowd=True, areas=False):
    pm, gm, fields = [], [], ([], [], [], [], [])
    for b in range(B):
        h, w = (int(v) for v in rng.integers(1, 40, 2))
        if aligned and b % 2:
            h, w = 16, 16 * int(rng.integers(1, 30))
        d, g = int(rng.integers(0, 150)), int(rng.integers(0, 80))
        pm.append(torch.zeros((d, h, w), dtype=torch.bool))
        gm.append(torch.zeros((g, h, w), dtype=torch.bool))
        wide = rng.random(4) < 0.5
        fields[0].append(torch.zeros(d, dtype=torch.int64 if wide[0] else torch.int32))
        fields[1].append(torch.zeros(d, dtype=torch.float64 if wide[1] else torch.float32))
        fields[2].append(torch.zeros(g, dtype=torch.int64 if wide[2] else torch.int32))
        fields[3].append(torch.zeros(g, dtype=torch.bool))
        fields[4].append(torch.zeros(g, dtype=torch.float64 if wide[3] else torch.float32))
    return (InstanceBatch(pm, fields[0], fields[1]),
            InstanceBatch(tuple(gm), fields[2], crowd=fields[3] if crowd else None,
                          areas=tuple(fields[4]) if areas else None))


@pytest.mark.parametrize("seed", range(6))
def test_instance_tables_are_the_python_paths(seed, host, on_cpu):
    from panoptic_evaluator_gb300 import _batch, instance, tuning
    rng = np.random.default_rng(seed)
    B = int(rng.integers(1, 12))
    prediction, target = _instances(rng, B, aligned=seed % 2, crowd=seed % 3 > 0, areas=seed % 2 == 0)
    raw, bounds_at, blocks_at, maps_at, rows_at, n_blocks, chunks, ranges = host.instance_tables(
        prediction, target, tuning.contract_costs(), _batch.CONTRACT_TMA_COST)
    words = np.frombuffer(raw, np.int64)
    # The table of InstanceEvaluator's Python path.
    shapes = np.array([tuple(m.shape) for m in prediction.masks])
    dets, gts = shapes[:, 0], np.array([m.shape[0] for m in target.masks])
    pixels = shapes[:, 1] * shapes[:, 2]
    table = _batch.DescTable(B)
    d = table.desc
    pm, gm = (np.array([m.data_ptr() for m in x.masks], np.int64) for x in (prediction, target))
    pairs, steps = dets * gts, (pixels + _batch.INST_CHUNK - 1) // _batch.INST_CHUNK
    for field, value in ((_batch.PIXELS, pixels), (_batch.MASK_STRIDE, pixels), (_batch.MASKS, pm),
                         (_batch.TARGET, gm), (_batch.D, dets), (_batch.G, gts),
                         (_batch.DET_BEGIN, np.cumsum(dets) - dets), (_batch.SLOT_BEGIN, np.cumsum(gts) - gts),
                         (_batch.DPAIR_BEGIN, np.cumsum(pairs) - pairs),
                         (_batch.CHUNK_BEGIN, np.cumsum(steps) - steps),
                         (_batch.FLAGS, instance.mask_flags(pm, gm, pixels))):
        d[:, field] = value
    plan = instance.contract_plan(table, dets, gts, pixels, torch.device("cpu"))
    table.finish(_batch.Scratch("cpu"), bounds=plan.extra)
    expected = table.device.numpy()
    head = table.extra_offset()
    assert bounds_at == head
    np.testing.assert_array_equal(words[:head], expected[:head])
    assert (n_blocks, chunks, ranges) == (len(plan.blocks), plan.total_chunks, plan.ctas)
    np.testing.assert_array_equal(words[blocks_at: blocks_at + 4 * n_blocks].reshape(-1, 4), plan.blocks)
    np.testing.assert_array_equal(words[bounds_at: bounds_at + ranges + 1],
                                  plan.extra[plan.blocks.size: plan.blocks.size + ranges + 1])
    assert (maps_at >= 0) == (plan.maps_at >= 0)
    if maps_at >= 0:
        np.testing.assert_array_equal(words[maps_at: maps_at + 32 * B],
                                      plan.extra[plan.maps_at: plan.maps_at + 32 * B])
    np.testing.assert_array_equal(words[rows_at: rows_at + 6 * B].reshape(B, 6),
                                  instance.gather_rows(prediction, target, B))


@pytest.mark.parametrize("seed", range(4))
def test_combined_tables_are_the_python_paths(seed, host, on_cpu, monkeypatch):
    from panoptic_evaluator_gb300 import _batch, combined
    rng = np.random.default_rng(seed)
    B, H, W, S, P = int(rng.integers(1, 7)), *(int(v) for v in rng.integers(1, 50, 2)), 9, 12
    if seed % 2:
        H = W = 32
    maps, pred = (torch.zeros((B, H, W), dtype=torch.int32) for _ in range(2))
    gc, pc = torch.zeros((B, S), dtype=torch.int32), torch.zeros((B, P), dtype=torch.int32)
    crowd = torch.zeros((B, S), dtype=torch.bool)
    n = [int(v) for v in rng.integers(0, 30, B)]
    masks = [torch.zeros((k, H, W), dtype=torch.bool) for k in n]
    classes = [torch.zeros(k, dtype=torch.int64 if rng.random() < 0.5 else torch.int32) for k in n]
    scores = [torch.zeros(k, dtype=torch.float64 if rng.random() < 0.5 else torch.float32) for k in n]
    raw, chunks = host.combined_tables(PanopticBatch(pred, pc), InstanceBatch(masks, classes, scores),
                                       PanopticBatch(maps, gc, crowd))
    words = np.frombuffer(raw, np.int64)
    seen = []
    monkeypatch.setattr(combined, "launch", lambda ev, table, *rest: seen.append(table))
    ev = SimpleNamespace(instance=SimpleNamespace(_scratch=_batch.Scratch("cpu")), device=torch.device("cpu"))
    combined.run_batch(ev, maps, pred, gc, pc, crowd, masks, classes, scores, None, [H * W] * B)
    table, = seen
    head = table.extra_offset()
    np.testing.assert_array_equal(words[:head], table.device.numpy()[:head])
    assert chunks == table.total_chunks
    rows = words[head:].reshape(B, 6)
    for b in range(B):
        assert list(rows[b, :3]) == [classes[b].data_ptr(), scores[b].data_ptr(), gc[b].data_ptr()]
        assert rows[b, 5] == (classes[b].dtype == torch.int64) + 2 * (scores[b].dtype == torch.float64)


@pytest.mark.parametrize("points", [None, (), (0,), (1, 3), (0, 2)])
def test_prefix_tables_are_the_python_paths(points, host, on_cpu, monkeypatch):
    from panoptic_evaluator_gb300 import prefix as PF
    captured = []
    n = [5, 3, 8] if points else [5, 0, 8]
    for B, H, W in ((3, 7, 9), (3, 16, 16), (1, 4, 5)):
        maps = torch.zeros((B, H, W), dtype=torch.int32)
        gc, crowd = torch.zeros((B, 4), dtype=torch.int32), torch.zeros((B, 4), dtype=torch.bool)
        masks = [torch.zeros((k, H, W), dtype=torch.bool) for k in n[:B]]
        classes = [torch.zeros(k, dtype=torch.int32) for k in n[:B]]
        raw, descs_at, steps_at, rows = host.prefix_tables(InstanceBatch(masks, classes),
                                                           PanopticBatch(maps, gc, crowd), 11, (0.5, 0.75), points)
        lists = [list(points) if points is not None else (list(range(1, k + 1)) if k else [0]) for k in n[:B]]
        with monkeypatch.context() as patch:
            patch.setattr(N, "call", lambda name, *args: captured.append(args) or 0)
            kept = PF.run_prefixes(maps, gc, crowd, masks, classes, 11, torch.ones(11, dtype=torch.uint8), (0.5, 0.75),
                                   lists, False)
        args = captured.pop()
        assert rows == args[3] == sum(map(len, lists))
        assert list(np.frombuffer(raw, np.float64, 2)) == list(kept[3])
        desc = np.ctypeslib.as_array((ctypes.c_int64 * (B * PF.FIELDS)).from_address(args[0]))
        np.testing.assert_array_equal(np.frombuffer(raw, np.int64, B * PF.FIELDS, descs_at), desc)
        count = sum(k + 1 for k in n[:B])
        steps = np.ctypeslib.as_array((ctypes.c_int32 * count).from_address(args[7]))
        np.testing.assert_array_equal(np.frombuffer(raw, np.int32, count, steps_at), steps)


def test_forms_the_host_path_leaves_to_python(host):
    """Other dtypes, strides, containers, subclasses and fields: no tables, the Python path takes the call."""
    rng = np.random.default_rng(1)
    prediction, target = _instances(rng, 3, aligned=False)
    tables = lambda p, t: host.instance_tables(p, t, {}, 0.73)  # noqa: E731
    assert tables(prediction, target) is not None
    change = lambda batch, **f: InstanceBatch(**{**batch.__dict__, **f})  # noqa: E731
    assert tables(change(prediction, scores=[s.half() for s in prediction.scores]), target) is None
    assert tables(change(prediction, masks=[m.to(torch.uint8) for m in prediction.masks]), target) is None
    strided = [torch.zeros((m.shape[0], m.shape[1], 2 * m.shape[2]), dtype=torch.bool)[:, :, ::2] for m in target.masks]
    assert tables(prediction, change(target, masks=strided)) is None
    assert tables(change(prediction, masks=iter(prediction.masks)), target) is None
    assert tables(change(prediction, classes=prediction.classes[:2]), target) is None
    assert tables(change(prediction, scores=None), target) is None
    subclass = [m.as_subclass(torch.nn.Buffer) if hasattr(torch.nn, "Buffer") else torch.nn.Parameter(m, False)
                for m in prediction.masks]
    assert tables(change(prediction, masks=subclass), target) is None
    other = [torch.zeros((m.shape[0], m.shape[1] + 1, m.shape[2]), dtype=torch.bool) for m in target.masks]
    assert tables(prediction, change(target, masks=other)) is None
    assert tables(InstanceBatch([], [], []), InstanceBatch([], [])) is None


# ---- on the GPU ------------------------------------------------------------------------------------------


@contextlib.contextmanager
def python_path():
    """A replaced `call` sees every entry point, so the evaluators take the Python path."""
    original = N.call
    N.call = lambda name, *args: original(name, *args)
    try:
        yield
    finally:
        N.call = original


def both(run):
    """run() through the host path and through the Python path: results or the error each raised."""
    outcomes = []
    for path in (contextlib.nullcontext, python_path):
        with path():
            try:
                outcomes.append(run())
            except Exception as error:  # noqa: BLE001
                outcomes.append((type(error), str(error)))
    return outcomes


def same(a, b, path="result"):
    if isinstance(a, dict) or hasattr(a, "keys"):
        assert list(a) == list(b), path
        for key in a:
            same(a[key], b[key], f"{path}/{key}")
    elif isinstance(a, torch.Tensor):
        assert a.dtype == b.dtype and a.shape == b.shape and a.device == b.device, path
        if a.is_floating_point():  # class sums of several images are added in any order
            torch.testing.assert_close(a, b, rtol=1e-13, atol=1e-15, equal_nan=True, msg=lambda m: f"{path}: {m}")
        else:
            assert torch.equal(a, b), path
    elif isinstance(a, (list, tuple)) and not isinstance(a, str):
        assert len(a) == len(b), path
        for i, (x, y) in enumerate(zip(a, b)):
            same(x, y, f"{path}[{i}]")
    else:
        assert a == b, (path, a, b)


def _cuda(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _scene(seed, B=2, H=37, W=53, dets=(0, 25)):
    from panoptic_evaluator_gb300 import synthetic
    rng = np.random.default_rng(seed)
    images = [synthetic.segmentation_image(rng, H, W, 12, int(rng.integers(*dets)), num_classes=9, things=6)
              for _ in range(B)]
    stack = lambda key: _cuda(np.stack([getattr(i, key) for i in images]))  # noqa: E731
    target = PanopticBatch(stack("target"), stack("target_classes"), stack("crowd"))
    prediction = PanopticBatch(stack("pred"), stack("pred_classes"))
    detections = InstanceBatch([_cuda(i.det_masks) for i in images], [_cuda(i.det_classes) for i in images],
                               [_cuda(i.scores) for i in images])
    return images, prediction, detections, target


def _forms(batch, form):
    change = lambda **f: type(batch)(**{**batch.__dict__, **f})  # noqa: E731
    if form == "tuples":
        return change(masks=tuple(batch.masks), classes=tuple(batch.classes))
    if form == "wide":
        return change(classes=[c.long() for c in batch.classes], scores=[s.double() for s in batch.scores])
    if form == "narrow":
        return change(classes=[c.int() for c in batch.classes])
    if form == "half":
        return change(scores=[s.half() for s in batch.scores])
    if form == "strided":
        return change(masks=[torch.stack((m, m), -1)[..., 0] for m in batch.masks])
    if form == "empty masks":
        return change(masks=[torch.zeros_like(m) for m in batch.masks])
    if form == "bad class":
        return change(classes=[c + 100 for c in batch.classes])
    if form == "nan score":
        return change(scores=[s * float("nan") for s in batch.scores])
    if form == "short field":
        return change(scores=[s[1:] for s in batch.scores])
    if form == "wrong dtype":
        return change(masks=[m.to(torch.uint8) for m in batch.masks])
    if form == "offset":
        return change(masks=[torch.cat((m.flatten(), m.flatten()[:3]))[: m.numel()].view(m.shape) if not m.numel() else
                             torch.cat((m.flatten()[:3], m.flatten()))[3:].view(m.shape) for m in batch.masks])
    return batch


FORMS = ("plain", "tuples", "wide", "narrow", "half", "strided", "offset", "empty masks", "bad class", "nan score",
         "short field", "wrong dtype")


@pytest.mark.gpu
@pytest.mark.parametrize("validate", (True, False))
@pytest.mark.parametrize("form", FORMS)
def test_combined_and_instance_calls_agree(form, validate):
    import panoptic_evaluator_gb300 as pe
    images, prediction, detections, target = _scene(7)
    batch = _forms(detections, form)
    masks = [torch.stack([_cuda(i.target == s) for s in range(1, 6)]) for i in images]
    labels = [torch.arange(5, device="cuda") % 6 for _ in images]

    def combined():
        ev = pe.SegmentationEvaluator(9, isthing=[True] * 6 + [False] * 3, validate=validate)
        for _ in range(2):
            ev.update(prediction, batch, target)
        first = ev.compute()
        ev.reset()
        return first, ev.update(prediction, batch, target).compute(), ev.state_dict()

    def instance(areas, crowd):
        ev = pe.InstanceEvaluator(9, validate=validate)
        truth = InstanceBatch(masks, labels, crowd=[c % 2 > 0 for c in labels] if crowd else None,
                              areas=[m.flatten(1).sum(1) * 0.5 for m in masks] if areas else None)
        for _ in range(2):
            ev.update(batch, truth)
        first = ev.compute()
        ev.reset()
        return first, ev.update(batch, truth).compute(), ev.state_dict()

    same(*both(combined))
    same(*both(lambda: instance(False, False)))
    same(*both(lambda: instance(True, True)))


@pytest.mark.gpu
@pytest.mark.parametrize("validate", (True, False))
@pytest.mark.parametrize("fault", ("none", "no crowd", "int64 map", "short classes", "bad slot", "bad class",
                                   "ghost class", "other shape", "transposed", "no images"))
def test_panoptic_and_prefix_calls_agree(fault, validate):
    import panoptic_evaluator_gb300 as pe
    _, prediction, detections, target = _scene(11, dets=(4, 9))
    maps, classes, crowd = target.segment_map.clone(), target.classes.clone(), target.crowd
    if fault == "no crowd":
        crowd = None
    elif fault == "int64 map":
        maps = maps.long()
    elif fault == "short classes":
        classes = classes[:1]
    elif fault == "bad slot":
        maps[0, 0, 0] = 1000
    elif fault == "bad class":
        classes[0, 1] = 99
    elif fault == "ghost class":
        classes[0, -1] = 3 if int(classes[0, -1]) < 0 else -1
    elif fault == "other shape":
        maps = maps[:, :-1].contiguous()
    elif fault == "transposed":
        maps = maps.transpose(1, 2).contiguous().transpose(1, 2)
    if fault == "no images":
        maps, classes, crowd = maps[:0], classes[:0], crowd[:0]
        prediction = PanopticBatch(prediction.segment_map[:0], prediction.classes[:0])
        detections = InstanceBatch([], [], [])
    truth = PanopticBatch(maps, classes, crowd)
    if not validate and fault == "bad class":
        return  # unchecked classes index the accumulators: not a valid call

    def update():
        ev = pe.PanopticEvaluator(9, isthing=[True] * 6 + [False] * 3, validate=validate)
        for _ in range(2):
            ev.update(prediction, truth)
        first = ev.compute()
        ev.reset()
        return first, ev.update(prediction, truth).compute(), ev.state_dict()

    def prefixes(**options):
        out = pe.segmentation_prefixes(InstanceBatch(detections.masks, [c.int() for c in detections.classes]), truth, 9,
                                       isthing=[True] * 6 + [False] * 3, validate=validate, **options)
        return [[dict(s) for s in image] for image in out]

    same(*both(update))
    same(*both(lambda: pe.panoptic_quality(prediction, truth, 9, validate=validate)))
    same(*both(lambda: pe.panoptic_quality(prediction, truth, 9, validate=validate, return_stats=True)))
    same(*both(prefixes))
    same(*both(lambda: prefixes(checkpoints=(0, 2, 4), iou_thresholds=(0.5, 0.6, 1))))
    same(*both(lambda: prefixes(checkpoints=())))
    same(*both(lambda: prefixes(checkpoints=(50,))))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ("rgb", "int32", "int64"))
@pytest.mark.parametrize("fault", ("none", "numpy ids", "duplicate id", "unknown category", "absent segment", "bool id",
                                   "no segments", "repeated category", "generator"))
def test_coco_tables_agree(kind, fault):
    rng = np.random.default_rng(3)
    ids = np.array([[0, 7, 70000, 300], [0, 9, 65535, 16777215]])
    slots = rng.integers(0, 4, (2, 11, 13))
    maps = np.take_along_axis(ids, slots.reshape(2, -1), 1).reshape(slots.shape)
    if kind == "rgb":
        maps = np.stack((maps % 256, maps // 256 % 256, maps // 65536), -1).astype(np.uint8)
    else:
        maps = maps.astype(kind)
    info = [[dict(id=int(i), category_id=int(20 + k), **({"iscrowd": 1} if k == 2 else {}))
             for k, i in enumerate(row[1:])] for row in ids]
    categories = [22, 20, 21, 23]
    if fault == "numpy ids":
        info = [[dict(e, id=np.int64(e["id"])) for e in row] for row in info]
    elif fault == "duplicate id":
        info[1][2]["id"] = info[1][0]["id"]
    elif fault == "unknown category":
        info[0][1]["category_id"] = 99
    elif fault == "absent segment":
        info[1] = info[1][:2]
    elif fault == "bool id":
        info[0][0]["id"] = True
    elif fault == "no segments":
        info, maps = [[], []], np.zeros_like(maps)
    elif fault == "repeated category":
        categories = [22, 20, 21, 20]
    device = _cuda(maps)

    def build():
        given = (c for c in categories) if fault == "generator" else categories
        batch = PanopticBatch.from_coco(device, info, given)
        return batch.segment_map, batch.classes, batch.crowd, batch.lookup_ids

    same(*both(build))


@pytest.mark.gpu
def test_uneven_images_agree_and_capture(tmp_path):
    import panoptic_evaluator_gb300 as pe
    from panoptic_evaluator_gb300 import synthetic
    from panoptic_evaluator_gb300.ragged import SegmentationImages
    images = synthetic.segmentation_batch(seed=4, images=5, side=(20, 90), slots=(3, 20), dets=(0, 9))
    fields = ("target", "target_classes", "crowd", "pred", "pred_classes", "det_masks", "det_classes", "scores")
    areas = [np.linspace(10, 9000, len(i.target_classes)) for i in images]
    isthing = [c < 80 for c in range(133)]
    for extra in ((), (areas,)):
        arena = SegmentationImages(*[[getattr(i, f) for i in images] for f in fields], *extra)

        def run():
            ev = pe.SegmentationEvaluator(133, isthing=isthing)
            ev.update_images(arena).update_images(arena)
            return ev.compute(), ev.state_dict()

        same(*both(run))
    # A captured step (reset, update, compute) replays through the host path.
    ev = pe.SegmentationEvaluator(133, isthing=isthing, validate=False)
    step = lambda: (ev.reset(), ev.update_images(arena), ev.compute())[2]  # noqa: E731
    eager = {k: v.clone() for k, v in step()["instance"].items()}
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    same(dict(captured["instance"]), eager)


@pytest.mark.gpu
def test_other_streams_and_threads_get_their_own_results():
    import threading

    import panoptic_evaluator_gb300 as pe
    scenes = [_scene(20 + k, B=3, H=90, W=110) for k in range(4)]
    expected = []
    for _, prediction, detections, target in scenes:
        ev = pe.SegmentationEvaluator(9, isthing=[True] * 6 + [False] * 3)
        expected.append(ev.update(prediction, detections, target).compute())
    torch.cuda.synchronize()
    results, errors = [None] * len(scenes), []

    def work(k):
        try:
            _, prediction, detections, target = scenes[k]
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(20):
                    ev = pe.SegmentationEvaluator(9, isthing=[True] * 6 + [False] * 3)
                    results[k] = ev.update(prediction, detections, target).compute()
                    rewards = pe.panoptic_quality(prediction, target, 9)
                    del rewards
            stream.synchronize()
        except Exception as error:  # noqa: BLE001
            errors.append(error)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(scenes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for got, want in zip(results, expected):
        same(got, want)
