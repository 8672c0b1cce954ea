"""Mask intersections by streaming and by contraction, and the choice between them: exact counts either way.

Counts are integers, so every comparison is exact; the reference is a float64 product of 0/1 masks (sums below 2^53).
"""

import numpy as np
import pytest
import torch

from panoptic_evaluator_gb300 import _batch, instance
from panoptic_evaluator_gb300 import _native as N


def _limit(dets, gts, pixels, sms=152):
    arrays = [np.ascontiguousarray(a, np.int64) for a in (dets, gts, pixels)]
    return N.call("pe_stream_limit", *(a.ctypes.data for a in arrays), None, len(arrays[0]), sms)


def test_small_batches_are_contracted_and_large_ones_may_stream():
    assert _limit([], [], []) == 0
    assert _limit([100], [8], [640 * 480]) == 0
    assert _limit([0] * 64, [0] * 64, [640 * 480] * 64) == 0
    few, many = _limit([100] * 16, [8] * 16, [410_000] * 16), _limit([100] * 64, [8] * 64, [410_000] * 64)
    assert 0 < few < many


def _masks(n, h, w, density, generator):
    if density == "none":
        return torch.zeros((n, h, w), dtype=torch.bool, device="cuda")
    if density == "full":
        return torch.ones((n, h, w), dtype=torch.bool, device="cuda")
    if density == "ends":  # the first and last pixel only
        m = torch.zeros((n, h * w), dtype=torch.bool, device="cuda")
        m[:, 0] = m[:, -1] = True
        return m.view(n, h, w)
    return torch.rand((n, h, w), device="cuda", generator=generator) < density


def _count(pm, gm, limit, monkeypatch, estimate=None):
    """pairwise_intersections through pe_inst_intersect; limit None: the batch's own."""
    def overlaps(scratch, table, dets, gts, pixels, chunks, order, pc, gc, inter, inter_len, pa, pa_len, ga, ga_len,
                 error, stream, method=None, plan=None):
        steps = -(-pixels // 4096)
        table.descs.view(len(dets), -1)[:, _batch.CHUNK_BEGIN] = torch.from_numpy(np.cumsum(steps) - steps).cuda()
        blocks, bounds, maps = plan.pointers(table)
        work = torch.full((8 * len(dets) + 1,), -1, dtype=torch.int64, device="cuda")
        N.call("pe_inst_intersect", table.descs.data_ptr(), len(dets), int(steps.sum()), blocks, len(plan.blocks),
               plan.total_chunks, bounds, plan.ctas, order.data_ptr(), inter.data_ptr(), inter_len, pa.data_ptr(),
               pa_len, ga.data_ptr(), ga_len, maps,
               max(_limit(dets, gts, pixels), 1) if limit is None else limit, work.data_ptr(), error.data_ptr(), stream)
        if estimate is not None:
            estimate.append(int(work[:-1].sum()))
    monkeypatch.setattr(instance, "overlaps", overlaps)
    return instance.pairwise_intersections(pm, gm)


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [-1, 2**62, None])
@pytest.mark.parametrize("images", [
    [(1, 1, 1, 1, "full")], [(3, 2, 5, 7, 0.5)], [(4, 3, 16, 16, "ends")], [(5, 0, 33, 31, 0.3), (0, 4, 20, 9, 0.3)],
    [(127, 63, 64, 64, 0.2)], [(128, 64, 63, 65, 0.2)], [(130, 130, 61, 67, 0.05)], [(9, 40, 64, 65, "full")],
    [(6, 33, 127, 33, 0.5), (7, 9, 64, 512, 0.01), (2, 2, 4, 3, "none"), (100, 8, 37, 111, "ends")],
    [(20, 12, 641, 13, 0.001), (20, 12, 4096, 1, "ends"), (20, 12, 4097, 1, "ends"), (3, 70, 513, 3, "full")],
])
def test_both_ways_count_every_pair(images, limit, monkeypatch):
    generator = torch.Generator("cuda").manual_seed(len(images) * 31 + images[0][0])
    pm = [_masks(d, h, w, f, generator) for d, g, h, w, f in images]
    gm = [_masks(g, h, w, f, generator) for d, g, h, w, f in images]
    for p, g, (inter, pa, ga) in zip(pm, gm, _count(pm, gm, limit, monkeypatch)):
        a, b = p.flatten(1).double(), g.flatten(1).double()
        assert torch.equal(inter, (a @ b.T).long())
        assert torch.equal(pa, a.sum(1).long()) and torch.equal(ga, b.sum(1).long())


@pytest.mark.gpu
@pytest.mark.parametrize("density, streamed", [(0.0002, True), (0.5, False)])
def test_the_masks_decide(density, streamed, monkeypatch):
    """A batch above the size limit: either way gives the evaluator's counts, and only one of the kernels works."""
    generator = torch.Generator("cuda").manual_seed(5)
    pm = [_masks(40, 511, 513, density, generator) for _ in range(40)]
    gm = [_masks(70, 511, 513, density, generator) for _ in range(40)]
    estimate = []
    chosen = _count(pm, gm, None, monkeypatch, estimate)
    assert (estimate[0] <= _limit([40] * 40, [70] * 40, [511 * 513] * 40)) == streamed
    for other in (-1, 2**62):
        for x, y in zip(chosen, _count(pm, gm, other, monkeypatch)):
            assert all(torch.equal(i, j) for i, j in zip(x, y))


@pytest.mark.gpu
@pytest.mark.parametrize("pixels", [(700, 500), (1117, 1201)])
@pytest.mark.parametrize("dets, gts", [(0, 3), (1, 1), (16, 2), (17, 64), (130, 5)])
def test_the_last_chunks_in_parts(pixels, dets, gts, monkeypatch):
    """Fewer chunks of 4096 pixels than two CTAs per SM, and a few more: parts of 16 detections and more."""
    generator = torch.Generator("cuda").manual_seed(dets)
    pm, gm = [_masks(dets, *pixels, 0.01, generator)], [_masks(gts, *pixels, 0.01, generator)]
    (inter, pa, ga), = _count(pm, gm, 2**62, monkeypatch)
    a, b = pm[0].flatten(1).double(), gm[0].flatten(1).double()
    assert torch.equal(inter, (a @ b.T).long())
    assert torch.equal(pa, a.sum(1).long()) and torch.equal(ga, b.sum(1).long())
