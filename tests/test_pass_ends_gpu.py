"""The fused pass at an image's last pixels, mask rows at every byte offset.

Counts are integers and must equal a float64 product of the 0/1 masks (sums below 2^53); results of the joint
evaluator must be the oracle's.
"""

import numpy as np
import pytest
import torch

from helpers import assert_tree, cuda

pytestmark = pytest.mark.gpu

# Pixel counts around a lane's 16 pixels, a warp's 512, a half's 4096 and a chunk's 8192, and every count mod 16.
PIXELS = [1, 2, 15, 16, 17, 495, 503, 511, 512, 513, 4079, 4095, *range(4097, 4113), 8191, 8193, 12288 + 497, 187500]


def _at_offset(array, elements):
    """A contiguous device copy that starts `elements` elements into its allocation."""
    flat = torch.zeros(array.size + elements, dtype=torch.from_numpy(array[:0].ravel()).dtype, device="cuda")
    view = flat[elements:].view(array.shape)
    view.copy_(torch.from_numpy(array))
    return view


@pytest.mark.parametrize("counter", (True, False))
@pytest.mark.parametrize("dets, offsets", [(1, range(16)), (17, range(16)), (130, (0, 5))])
def test_masks_of_the_last_pixels_are_counted(dets, offsets, counter):
    """Masks of an image's last 1 to 16 pixels alone: nothing else of a mask leads a warp to them."""
    from panoptic_evaluator_gb300 import _batch as F
    from panoptic_evaluator_gb300 import _native as N
    slots = 3
    sizes = [(n, o) for n in PIXELS for o in offsets]
    maps, masks = [], []
    for b, (n, o) in enumerate(sizes):
        maps.append((torch.arange(n, device="cuda", dtype=torch.int32) + b) % slots)
        rows = torch.zeros(dets * n + o, dtype=torch.bool, device="cuda")[o:].view(dets, n)
        last = 1 + (torch.arange(dets, device="cuda") + b // len(offsets)) % 16
        rows[:] = torch.arange(n, device="cuda") >= n - last[:, None]
        masks.append(rows)
    pixels = np.array([n for n, _ in sizes], np.int64)
    index = np.arange(len(sizes), dtype=np.int64)
    table = F.DescTable(len(sizes))
    d = table.desc
    d[:, F.TARGET] = d[:, F.PRED] = [m.data_ptr() for m in maps]
    d[:, F.MASKS] = [m.data_ptr() for m in masks]
    d[:, F.PIXELS] = d[:, F.MASK_STRIDE] = pixels
    chunks = -(-pixels // F.SEG_CHUNK)
    d[:, F.CHUNK_BEGIN] = np.cumsum(chunks) - chunks
    d[:, F.DET_BEGIN] = dets * index
    d[:, F.SLOT_BEGIN] = d[:, F.PSLOT_BEGIN] = slots * index
    d[:, F.PAIR_BEGIN] = slots * slots * index
    d[:, F.DPAIR_BEGIN] = dets * slots * index
    d[:, F.D], d[:, F.G], d[:, F.P] = dets, slots, slots
    table.finish(F.Scratch("cuda"))
    order = torch.arange(dets, device="cuda").repeat(len(sizes))
    pairs = torch.full((len(sizes), slots, slots), 7, dtype=torch.int32, device="cuda")
    counts = torch.full((len(sizes), dets, slots), 7, dtype=torch.int32, device="cuda")
    error = torch.zeros(1, dtype=torch.int32, device="cuda")
    schedule = torch.full((1,), 7, dtype=torch.int64, device="cuda") if counter else None
    N.call("pe_seg_pass", table.descs.data_ptr(), len(sizes), int(chunks.sum()), order.data_ptr(), pairs.data_ptr(),
           pairs.numel(), counts.data_ptr(), counts.numel(), slots * slots, dets * slots, 2, None, 0, N.ptr(schedule),
           error.data_ptr(), N.stream_handle(error.device))
    assert int(error) == 0
    for b, size in enumerate(sizes):
        on_slot = torch.nn.functional.one_hot(maps[b].long(), slots).double()
        assert torch.equal(counts[b].long(), (masks[b].double() @ on_slot).long()), size
        assert torch.equal(pairs[b].long(), torch.diag(on_slot.sum(0)).long()), size


@pytest.mark.parametrize("validate", (False, True))
@pytest.mark.parametrize("offset", (0, 3, 8))
@pytest.mark.parametrize("dets", (1, 17, 130))
@pytest.mark.parametrize("hw", [(375, 500), (479, 641), (37, 53), (3, 641)])
def test_objects_in_the_last_corner(hw, dets, offset, validate):
    import panoptic_evaluator_gb300 as pe
    from oracle import combined as ocomb
    rng = np.random.default_rng(hw[1] + dets + offset)
    h, w = hw
    n = h * w
    gt = np.full((2, h, w), 3, np.int32)
    gt[:, 0, :w // 2] = 0
    gt[:, :, -2:] = 2
    masks = []
    for b in range(2):
        last = int(rng.integers(1, 16))
        gt[b].reshape(-1)[n - last:] = 1
        rows = np.zeros((dets, n), bool)
        for i in range(dets):
            kind = i % 4
            if kind == 0:
                rows[i, n - (last if i == 0 else int(rng.integers(1, 16))):] = True
            elif kind == 1:
                rows[i].reshape(h, w)[-min(h, 40):, -2:] = True
            elif kind == 2:
                rows[i, -1] = True
            else:
                rows[i].reshape(h, w)[-8:, -8:] = True
        masks.append(rows.reshape(dets, h, w))
    gc = np.array([[-1, 0, 1, 2]] * 2, np.int32)
    crowd = np.zeros((2, 4), bool)
    labels = [np.arange(dets, dtype=np.int64) % 2 for _ in range(2)]
    scores = [np.concatenate(([2.0], rng.random(dets - 1))).astype(np.float32) for _ in range(2)]
    isthing = [True, True, False]
    oracle = ocomb.SegmentationOracle(3, isthing)
    oracle.update(gt, gc, masks, labels, scores, gt, gc, crowd)
    joint = pe.SegmentationEvaluator(3, isthing=isthing, validate=validate)
    joint.update(pe.PanopticBatch(cuda(gt), cuda(gc)),
                 pe.InstanceBatch([_at_offset(m, offset) for m in masks], [cuda(x) for x in labels],
                                  [cuda(s) for s in scores]),
                 pe.PanopticBatch(cuda(gt), cuda(gc), cuda(crowd)))
    assert_tree(joint.compute(), oracle.compute())
