"""Generation-order matching at the edges of its split: classes over several CTAs, chains of a thread or of a warp.

Integers must equal the oracle's exactly; precision and recall are single FP64 quotients of them (1e-12).
"""

import numpy as np
import pytest
import torch

from helpers import cuda
from oracle import prefix as opre

pytestmark = pytest.mark.gpu

# images, masks, slots, classes, IoU thresholds
CASES = [
    (1, 1, 2, 1, (0.5,)),
    (2, 0, 5, 3, (0.5, 0.75)),                        # no masks
    (1, 40, 41, 1, (0.05, 0.5, 0.75)),                # one class: a warp's chain, targets over two used words
    (2, 33, 100, 3, (0.3, 0.5)),                      # warps' chains whose used words meet
    (3, 64, 9, 1, (0.1, 0.5, 0.9)),                   # nine slots: over the serial slots and the pairs
    (3, 14, 9, 1, (0.1, 0.5, 0.9)),                   # nine slots, few enough pairs for a thread
    (2, 64, 101, 133, (0.5, 0.75)),                   # nine CTAs for an image's classes
    (1, 20, 30, 17, tuple(0.05 * k for k in range(1, 20))),  # more (threshold, class) chains than threads' warps
    (1, 150, 120, 1, (0.25, 0.5)),                    # more IoUs than shared memory has room for
    (160, 4, 12, 40, (0.5,)),                         # more images than SMs
]


@pytest.mark.parametrize("images, masks, slots, classes, thresholds", CASES)
def test_matching_follows_the_oracle(images, masks, slots, classes, thresholds):
    import panoptic_evaluator_gb300 as pe
    rng = np.random.default_rng(images + 7 * masks + slots)
    h, w = 16, 8 * slots
    gt = np.broadcast_to((np.arange(w) // 8).astype(np.int32), (images, h, w)).copy()
    gc = rng.integers(0, classes, (images, slots)).astype(np.int32)
    gc[:, 0] = -1
    crowd = (rng.random((images, slots)) < 0.1) & (gc >= 0)
    isthing = np.arange(classes) < max(1, classes * 3 // 4)
    drawn, labels = [], []
    for b in range(images):
        of = rng.integers(1, slots, masks)
        keep = rng.choice((0.3, 0.6, 0.8, 1.0), masks)  # equal IoUs among the masks of full height and the others
        rows = np.arange(h)[None, :, None] < np.ceil(keep * h)[:, None, None]
        wide = rng.integers(0, 3, masks)[:, None, None]  # up to two columns of the next slot
        column = np.arange(w)[None, None]
        left = 8 * of[:, None, None]
        drawn.append((column >= left) & (column < left + 8 + wide) & rows)
        labels.append(np.where(rng.random(masks) < 0.8, gc[b, of], rng.integers(0, classes, masks)).astype(np.int32))
    points = sorted({0, masks // 3, masks})
    result = pe.segmentation_prefixes(
        pe.InstanceBatch([cuda(m) for m in drawn], [cuda(c) for c in labels]),
        pe.PanopticBatch(cuda(gt), cuda(gc), cuda(crowd)), classes, isthing=isthing.tolist(), checkpoints=points,
        iou_thresholds=thresholds)
    expected = opre.segmentation_prefixes(drawn, labels, gt, gc, crowd, classes, isthing=isthing.tolist(),
                                          checkpoints=points, iou_thresholds=thresholds)
    for got, want in zip(result, expected, strict=True):
        for g, e in zip(got, want, strict=True):
            for key in ("tp", "fp", "fn"):
                np.testing.assert_array_equal(g["instance"][key].cpu().numpy(), e["instance"][key], err_msg=key)
                np.testing.assert_array_equal(g[key].cpu().numpy(), e[key], err_msg=key)
            for key in ("precision", "recall"):
                np.testing.assert_allclose(g["instance"][key].cpu().numpy(), e["instance"][key], rtol=0, atol=1e-12)
