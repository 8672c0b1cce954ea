"""Scoring kernels at the edges of their tiles: histogram alignment, entry lists, column blocks, class clusters.

Integers must equal the oracle's exactly; FP64 values agree within 1e-12 (sums of at most a few
thousand IoUs in (0.5, 1], each correctly rounded, averaged over the classes).
"""

import numpy as np
import pytest
import torch

from helpers import assert_tree
from oracle import panoptic as opan

pytestmark = pytest.mark.gpu

# B, H, W, G, P, classes, share of pixels whose prediction follows the target
SHAPES = [
    (2, 150, 150, 90, 110, 20, 0.6),   # more nonzero pairs than the entry list holds
    (1, 61, 67, 5, 1500, 3, 0.7),      # more column blocks than warps
    (1, 64, 64, 1500, 4, 70, 0.9),     # more targets than predictions, a cluster of CTAs per summary
    (3, 41, 43, 33, 45, 257, 0.9),     # odd pixel count: images start off the 16-byte grid; two column tiles
    (2, 1, 3, 2, 2, 64, 1.0),          # fewer pixels than one load
    (1, 1, 1, 1, 1, 1, 1.0),
    (5, 64, 65, 31, 32, 63, 0.95),
    (2, 127, 129, 33, 64, 133, 0.97),
]


def _arrays(seed, B, H, W, G, P, C, follow, consistent):
    rng = np.random.default_rng(seed)
    gt = (np.arange(H)[None, :, None] * 7 // max(1, H) * 5 + np.arange(W)[None, None, :] // 3 + rng.integers(0, G, (B, 1, 1)))
    gt = np.where(rng.random((B, H, W)) < 0.9, gt % G, rng.integers(0, G, (B, H, W))).astype(np.int32)
    pred = np.where(rng.random((B, H, W)) < follow, gt % P, rng.integers(0, P, (B, H, W))).astype(np.int32)
    gc = rng.integers(-1, C, (B, G)).astype(np.int32)
    pc = np.where(np.arange(P) < G, gc[:, np.minimum(np.arange(P), G - 1)], rng.integers(-1, C, (B, P))).astype(np.int32)
    if consistent:
        for classes, maps in ((gc, gt), (pc, pred)):
            present = np.stack([np.bincount(m.ravel(), minlength=classes.shape[1]) > 0 for m in maps])
            classes[:] = np.where(present, np.maximum(classes, 0), -1)
    gc[:, 0] = pc[:, 0] = -1
    crowd = (rng.random((B, G)) < 0.2) & (gc >= 0)
    return gt, gc, crowd, pred, pc


def _at_offset(array, elements):
    """A contiguous device copy that starts `elements` elements into its allocation."""
    flat = torch.zeros(array.size + elements, dtype=torch.from_numpy(array[:0].ravel()).dtype, device="cuda")
    view = flat[elements:].view(array.shape)
    view.copy_(torch.from_numpy(array))
    return view


@pytest.mark.parametrize("validate", (False, True))
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("offsets", ((0, 0), (1, 1), (2, 3)))
def test_update_compute_and_reward_match_the_oracle(shape, offsets, validate):
    import panoptic_evaluator_gb300 as pe
    C = shape[5]
    gt, gc, crowd, pred, pc = _arrays(11, *shape, consistent=validate)
    isthing = np.arange(C) < (C + 1) // 2
    oracle = opan.PanopticOracle(C, isthing, validate=validate)
    oracle.update(pred, pc, gt, gc, crowd)
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    target = pe.PanopticBatch(_at_offset(gt, offsets[0]), dev(gc), dev(crowd))
    prediction = pe.PanopticBatch(_at_offset(pred, offsets[1]), dev(pc))
    ev = pe.PanopticEvaluator(C, isthing=isthing.tolist(), validate=validate)
    ev.update(prediction, target)
    assert_tree(ev.compute(), oracle.compute())
    want = opan.panoptic_quality(pred, pc, gt, gc, crowd, C, validate_inputs=validate)
    got = pe.panoptic_quality(prediction, target, C, validate=validate)
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-12
    stats = pe.panoptic_quality(prediction, target, C, validate=validate, return_stats=True).cpu().numpy()
    expected = opan.panoptic_quality(pred, pc, gt, gc, crowd, C, validate_inputs=validate, return_stats=True)
    np.testing.assert_array_equal(stats[..., 1:], expected[..., 1:])
    assert np.abs(stats[..., 0] - expected[..., 0]).max() <= 1e-12


def test_an_unvalidated_void_class_adds_both_matches():
    """Slot 0 given a class (accepted without validation): its match and a segment's both count, as in the oracle."""
    import panoptic_evaluator_gb300 as pe
    gt = np.array([[[0, 0, 1, 1, 1, 2]]], np.int32)
    pred = np.array([[[1, 1, 1, 1, 1, 2]]], np.int32)
    gc, pc = np.array([[0, 0, 1]], np.int32), np.array([[-1, 0, 1]], np.int32)
    crowd = np.zeros((1, 3), bool)
    oracle = opan.PanopticOracle(2, [True, False], validate=False)
    oracle.update(pred, pc, gt, gc, crowd)
    ev = pe.PanopticEvaluator(2, isthing=[True, False], validate=False)
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    ev.update(pe.PanopticBatch(dev(pred), dev(pc)), pe.PanopticBatch(dev(gt), dev(gc), dev(crowd)))
    assert_tree(ev.compute(), oracle.compute())


def test_out_of_range_slots_are_reported_and_not_counted():
    import panoptic_evaluator_gb300 as pe
    gt = np.zeros((1, 5, 9), np.int32)
    gt[0, 2, 3] = 4  # capacity is 4 slots
    pred = np.zeros_like(gt)
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    classes = np.full((1, 4), -1, np.int32)
    ev = pe.PanopticEvaluator(3)
    before = {k: v.clone() for k, v in ev.state_dict().items()}
    with pytest.raises(ValueError, match="unknown segment ID or a slot outside"):
        ev.update(pe.PanopticBatch(dev(pred), dev(classes)), pe.PanopticBatch(dev(gt), dev(classes)))
    assert all(torch.equal(v, before[k]) for k, v in ev.state_dict().items())


@pytest.mark.parametrize("validate", (False, True))
@pytest.mark.parametrize("images", (1, 7, 77, 160))
def test_detection_areas_beside_the_scoring(images, validate):
    """Few images leave SMs that sum detection areas in blocks of their own; more than SMs share their blocks."""
    import panoptic_evaluator_gb300 as pe
    from oracle import combined as ocomb
    from panoptic_evaluator_gb300 import synthetic
    from panoptic_evaluator_gb300.ragged import SegmentationImages
    batch = synthetic.segmentation_batch(seed=images, images=images, side=(20, 60), slots=(3, 60), dets=(0, 40))
    isthing = list(np.arange(133) < 80)
    oracle = ocomb.SegmentationOracle(133, isthing)
    for i in batch:
        oracle.update(i.pred[None], i.pred_classes[None], [i.det_masks], [i.det_classes], [i.scores], i.target[None],
                      i.target_classes[None], i.crowd[None])
    fields = ("target", "target_classes", "crowd", "pred", "pred_classes", "det_masks", "det_classes", "scores")
    joint = pe.SegmentationEvaluator(133, isthing=isthing, validate=validate)
    joint.update_images(SegmentationImages(*([getattr(i, f) for i in batch] for f in fields)))
    assert_tree(joint.compute(), oracle.compute())


@pytest.mark.parametrize("offset", (0, 1, 4, 15))
@pytest.mark.parametrize("size", (0, 1, 3, 15, 16, 17, 31, 4096, 1_000_003))
def test_zeroing_clears_the_span_and_nothing_beside_it(offset, size):
    from panoptic_evaluator_gb300 import _native as N
    data = torch.full((size + 64,), 7, dtype=torch.uint8, device="cuda")
    N.call("pe_zero", data.data_ptr() + offset, size, N.stream_handle(data.device))
    want = torch.full_like(data, 7)
    want[offset:offset + size] = 0
    assert torch.equal(data, want)


@pytest.mark.parametrize("dets", (0, 1, 16, 17, 33, 130))
def test_the_last_halves_of_the_pass_in_parts(dets):
    """More halves of 4096 pixels than two CTAs per SM: whole ones, then parts of 16 detections and more."""
    import panoptic_evaluator_gb300 as pe
    from oracle import combined as ocomb
    from panoptic_evaluator_gb300 import synthetic
    from panoptic_evaluator_gb300.ragged import SegmentationImages
    batch = synthetic.segmentation_batch(seed=dets, images=2, fixed_hw=(1009, 701), slots=(20, 40), dets=(dets, dets))
    isthing = list(np.arange(133) < 80)
    oracle = ocomb.SegmentationOracle(133, isthing)
    fields = ("target", "target_classes", "crowd", "pred", "pred_classes", "det_masks", "det_classes", "scores")
    for i in batch:
        oracle.update(i.pred[None], i.pred_classes[None], [i.det_masks], [i.det_classes], [i.scores], i.target[None],
                      i.target_classes[None], i.crowd[None])
    joint = pe.SegmentationEvaluator(133, isthing=isthing)
    joint.update_images(SegmentationImages(*([getattr(i, f) for i in batch] for f in fields)))
    assert_tree(joint.compute(), oracle.compute())


@pytest.mark.parametrize("shape", [
    (1, 150, 150, 150, 120, 20, 0.6),   # eight CTAs an image, a list that overflows
    (3, 127, 129, 6000, 3, 7, 0.9),     # hardly any columns
    (2, 64, 129, 3, 6000, 5, 0.9),      # fewer rows than CTAs: row 0 with the first
    (2, 64, 65, 5, 4000, 5, 0.9),
    (20, 61, 67, 140, 130, 33, 0.9),    # four CTAs an image
    (60, 41, 43, 135, 145, 15, 0.9),    # two
    (90, 41, 43, 135, 145, 15, 0.9),    # more images than pairs of SMs
])
def test_counts_shared_by_a_cluster(shape):
    import panoptic_evaluator_gb300 as pe
    C = shape[5]
    gt, gc, crowd, pred, pc = _arrays(13, *shape, consistent=False)
    isthing = np.arange(C) < (C + 1) // 2
    oracle = opan.PanopticOracle(C, isthing, validate=False)
    oracle.update(pred, pc, gt, gc, crowd)
    ev = pe.PanopticEvaluator(C, isthing=isthing, validate=False)
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    ev.update(pe.PanopticBatch(dev(pred), dev(pc)), pe.PanopticBatch(dev(gt), dev(gc), dev(crowd)))
    assert_tree(ev.compute(), oracle.compute())
