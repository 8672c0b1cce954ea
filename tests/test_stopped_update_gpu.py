"""Updates whose kernels gave up: a checked one raises and leaves the totals, an unchecked one makes the metrics NaN.

No wait runs out here: the error word gets the bit of a timeout before the kernels that read it.
"""

import numpy as np
import pytest
import torch

from panoptic_evaluator_gb300 import _native as N

pytestmark = pytest.mark.gpu

TIMEOUT, UNCHECKED, UNKNOWN = 1 << 30, 1 << 27, -2**40


def _inputs(images):
    import panoptic_evaluator_gb300 as pe
    maps = torch.zeros((images, 9, 31), dtype=torch.int32, device="cuda")
    maps[:, 2:5], maps[:, 5:] = 1, 2
    classes = torch.tensor([[-1, 0, 1]] * images, dtype=torch.int32, device="cuda")
    target = pe.PanopticBatch(maps, classes, torch.zeros((images, 3), dtype=torch.bool, device="cuda"))
    masks = [torch.stack((m == 1, m == 2, m > 0)) for m in maps]
    labels = [torch.tensor([0, 1, 0], device="cuda")] * images
    detections = pe.InstanceBatch(masks, labels, [torch.tensor([0.9, 0.8, 0.7], device="cuda")] * images)
    return target, detections, pe.InstanceBatch([m[:2] for m in masks], [x[:2] for x in labels])


def _timeout_before(entry, scratch, monkeypatch):
    call = N.call

    def with_timeout(name, *args):
        if name == entry:
            scratch.get("error", 1, torch.int32).fill_(TIMEOUT)
        return call(name, *args)
    monkeypatch.setattr(N, "call", with_timeout)


def _fill_records(store):
    """Memory of records to come, as an earlier user may have left it: first-ranked true positives."""
    store.reserve(1)
    store.ranks[store.n:].fill_(1)
    store.flags[store.n:].fill_(1)


def _all_nan(result):
    return all(bool(torch.isnan(v).all()) for v in result.values())


@pytest.mark.parametrize("validate", (False, True))
def test_instance_update(validate, monkeypatch):
    import panoptic_evaluator_gb300 as pe
    _, detections, target = _inputs(3)
    ev = pe.InstanceEvaluator(2, validate=validate)
    ev.update(detections, target)
    expected, state = ev.compute(), ev.state_dict()
    _fill_records(ev._store)
    with monkeypatch.context() as patch:
        _timeout_before("pe_inst_prepare", ev._scratch, patch)
        if validate:
            with pytest.raises(RuntimeError):
                ev.update(detections, target)
        else:
            ev.update(detections, target)
    if validate:
        assert all(torch.equal(v, state[k]) for k, v in ev.state_dict().items())
        return
    assert ev.num_records == 18 and not ev._store.ranks[9:18].any() and bool((ev._store.flags[9:18] == -1).all())
    assert _all_nan(ev.compute())
    ev.update(detections, target)
    assert _all_nan(ev.compute())
    ev.reset()
    ev.update(detections, target)
    assert all(torch.equal(v, expected[k]) for k, v in ev.compute().items())


@pytest.mark.parametrize("validate", (False, True))
@pytest.mark.parametrize("images", (1, 3, 200))
def test_joint_update(images, validate, monkeypatch):
    import panoptic_evaluator_gb300 as pe
    target, detections, _ = _inputs(images)
    ev = pe.SegmentationEvaluator(2, validate=validate)
    ev.update(target, detections, target)
    expected, state = ev.compute(), ev.state_dict()
    _fill_records(ev.instance._store)
    with monkeypatch.context() as patch:
        _timeout_before("pe_seg_score", ev.instance._scratch, patch)
        if validate:
            with pytest.raises((RuntimeError, ValueError)):
                ev.update(target, detections, target)
        else:
            ev.update(target, detections, target)
    if validate:
        assert all(torch.equal(v, state[k]) for k, v in ev.state_dict().items())
        return
    stopped = ev.compute()
    assert _all_nan(stopped["instance"])
    for name in ("All", "Things"):
        assert bool(torch.isnan(stopped[name]["pq"])) and bool(torch.isnan(stopped[name]["sq"]))
    assert bool(torch.isnan(stopped["miou"]))
    for name in ("tp", "fp", "fn", "confusion"):
        assert torch.equal(stopped[name], expected[name])
    ev.reset()
    ev.update(target, detections, target)
    result = ev.compute()
    assert torch.equal(result["miou"], expected["miou"])
    assert all(torch.equal(v, expected["instance"][k]) for k, v in result["instance"].items())
    assert all(torch.equal(result["All"][k], expected["All"][k]) for k in ("pq", "sq", "rq", "n"))


@pytest.mark.parametrize("entry, gate, unknown", [
    ("pe_inst_match", TIMEOUT, True), ("pe_inst_match", 1 << 28, True), ("pe_inst_match", 4, False),
    ("pe_seg_match", TIMEOUT, False), ("pe_seg_match", TIMEOUT | UNCHECKED, True), ("pe_seg_match", 4, False),
])
def test_gated_matching_defines_its_records(entry, gate, unknown):
    classes, dets = 3, (2, 0, 5)
    dev = lambda x, t: torch.as_tensor(np.asarray(x), dtype=t, device="cuda")  # noqa: E731
    total = sum(dets)
    area = torch.int64 if entry == "pe_inst_match" else torch.float64
    off = dev(np.concatenate(([0], np.cumsum(dets))), torch.int64)
    pairs, pair_off = dev([1] * total, torch.int32), off[:-1].contiguous()  # one target per image
    g_off = dev(range(4), torch.int64)
    pc, gc = dev([0] * total, torch.int32), dev([0] * 3, torch.int32)
    pa, ga, areas = dev([1] * total, area), dev([1] * 3, area), dev([1] * 3, torch.float64)
    crowd = dev([0] * 3, torch.uint8)
    flags, ranks = dev(np.full((total + 1, 40), 7), torch.int8), dev([7] * (total + 1), torch.int32)
    counts, word = dev(np.full((classes, 4), 5), torch.int64), dev([gate], torch.int32)
    N.call(entry, pairs.data_ptr(), pair_off.data_ptr(), off.data_ptr(), g_off.data_ptr(), 3, pc.data_ptr(),
           pa.data_ptr(), gc.data_ptr(), ga.data_ptr(), crowd.data_ptr(), areas.data_ptr(), classes, 1,
           flags.data_ptr(), 1, 40, ranks.data_ptr(), counts.data_ptr(), word.data_ptr(), None,
           N.stream_handle(word.device))
    assert ranks.tolist() == [0] * total + [7]
    assert bool((flags[:-1] == -1).all()) and bool((flags[-1] == 7).all())
    assert bool((counts == (UNKNOWN if unknown else 5)).all())


def test_prefixes(monkeypatch):
    """The void slot's pixel count (above 2^20) stands in for the error word of an owner pass that gave up."""
    import panoptic_evaluator_gb300 as pe
    maps = torch.zeros((1, 1025, 1100), dtype=torch.int32, device="cuda")
    maps[:, :30], maps[:, 30:60] = 1, 2
    classes = torch.tensor([[-1, 0, 70]], dtype=torch.int32, device="cuda")
    target = pe.PanopticBatch(maps, classes, torch.zeros((1, 3), dtype=torch.bool, device="cuda"))
    masks = pe.InstanceBatch([torch.stack((maps[0] == 1, maps[0] == 2))], [torch.tensor([0, 70], device="cuda")])
    expected, = pe.segmentation_prefixes(masks, target, 71, validate=False)
    call = N.call

    def with_timeout(name, *args):
        return call(name, *args[:-2], args[15], args[-1]) if name == "pe_prefix" else call(name, *args)
    monkeypatch.setattr(N, "call", with_timeout)
    stopped, = pe.segmentation_prefixes(masks, target, 71, validate=False)
    for now, then in zip(stopped, expected):
        assert not bool(torch.isnan(then["iou_sum"]).any()) and torch.equal(now["tp"], then["tp"])
        assert bool(torch.isnan(now["All"]["pq"])) and bool(torch.isnan(now["miou"]))
        assert bool(torch.isnan(now["iou_sum"]).all())
        assert bool(torch.isnan(now["instance"]["precision"]).all())
        assert bool(torch.isnan(now["instance"]["recall"]).all())
