"""Matching, sorting and accumulation at the edges of their lists and stages, against the oracle.

Match outcomes, ranks and counts are integers (exact); precision and recall are single correctly
rounded quotients of integers, the same in the oracle, so 1e-12 leaves room for nothing but a
different count.
"""

import numpy as np
import pytest
import torch

from oracle import instance as oinst


def test_integer_recall_thresholds_equal_the_floating_point_search():
    """t = ceil(np r / 100), one more where np r is a multiple of 100 and r / 100 rounds below r * 0.01."""
    r = np.arange(101, dtype=np.int64)
    threshold = r.astype(np.float64) * 0.01
    short = r.astype(np.float64) / 100.0 < threshold
    for positives in [*range(1, 1200), 4999, 5000, 12345, 99900, 10**6, 2**31 - 1, 10**12 + 300]:
        scaled = positives * r
        t = (scaled + 99) // 100
        t = t + ((t * 100 == scaled) & short)
        assert ((t / positives >= threshold) | (t > positives)).all()
        below = t > 0
        assert ((t[below] - 1) / positives < threshold[below]).all()


def _pairs(rng, D, G, kind):
    if kind == "same":  # near-identical masks: every pair is a candidate, many ties
        pairs = rng.integers(900, 1001, (D, G)) // 20 * 20
        return pairs, np.full(D, 1000.0), np.full(G, 1000.0)
    pa, ga = rng.integers(1, 12000, D).astype(np.float64), rng.integers(1, 12000, G).astype(np.float64)
    share = np.where(rng.random((D, G)) < (0.9 if kind == "sparse" else 0.4), 0.0, rng.uniform(0.5, 1.0, (D, G)))
    return (share * np.minimum(pa[:, None], ga[None])).astype(np.int64), pa, ga


@pytest.mark.gpu
@pytest.mark.parametrize("D, G, C, kind", [
    (1, 1, 1, "same"), (7, 0, 2, "same"), (0, 5, 2, "same"), (30, 33, 1, "same"),
    (120, 60, 2, "same"),       # more than 100 detections of a class, more candidates than the list holds
    (40, 130, 1, "dense"), (101, 31, 3, "dense"), (64, 32, 1, "sparse"), (200, 200, 9, "sparse"),
    (90, 600, 1, "sparse"),
])
def test_greedy_matching_equals_the_oracle(D, G, C, kind):
    from panoptic_evaluator_gb300 import _cuda_evaluator as native
    rng = np.random.default_rng(D * 1000 + G)
    pairs, pa, ga = _pairs(rng, D, G, kind)
    pc, gc = rng.integers(0, C, D).astype(np.int32), rng.integers(0, C, G).astype(np.int32)
    if D > 3:
        pc[::17] = C + 1  # outside the classes: never ranked
    crowd = rng.random(G) < 0.15
    areas = np.where(rng.random(G) < 0.5, ga, rng.choice([1024.0, 9216.0, 500.0, 20000.0], G))
    union = np.where(crowd[None], pa[:, None], pa[:, None] + ga[None] - pairs)
    status, ranks, counts = oinst.match_ious(pairs / np.maximum(union, 1), pc, gc, pa, crowd, areas, C)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    got = native.instance_match_histogram(dev(pairs.astype(np.int64)), dev(pc), dev(gc), dev(pa), dev(ga), dev(crowd),
                                          dev(areas), C)
    for value, want in zip(got, (status, ranks, counts)):
        np.testing.assert_array_equal(value.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [
    (0, 0), (1, 0, 2), (191, 192, 193), (511, 512, 513), (1023, 1024, 1025), (1500, 3, 700),
    (2700, 2700, 2792), (2700, 2700, 2793),  # the last records count every block scans, and the first grouped
    (9000, 40, 600, 1100),
])
def test_accumulation_equals_the_oracle(sizes):
    from panoptic_evaluator_gb300 import _cuda_evaluator as native
    rng = np.random.default_rng(sum(sizes) + len(sizes))
    C, n = len(sizes), sum(sizes)
    classes = rng.permutation(np.repeat(np.arange(C, dtype=np.int32), sizes)) if n else np.zeros(0, np.int32)
    ranks = rng.integers(0, 130, n).astype(np.int32)
    ranks[ranks > 100] = 0
    flags = rng.choice(np.array([-1, 0, 1], np.int8), (40, n), p=(0.2, 0.4, 0.4))
    counts = rng.choice([0, 1, 4, 50, 100, 200, 5000, 10000], (C, 4)).astype(np.int64)
    for c in range(C):  # a class has at least as many targets as matches
        for a in range(4):
            most = int((flags[10 * a:10 * a + 10, (classes == c) & (ranks > 0)] == 1).sum(1).max(initial=0))
            if counts[c, a]:
                counts[c, a] = max(counts[c, a], most)
    precision, recall = oinst.accumulate(classes, ranks, flags, counts)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    got = native.instance_compute(dev(classes), dev(ranks), dev(flags), dev(counts))
    assert np.abs(got[0].cpu().numpy() - precision).max() <= 1e-12
    assert np.abs(got[1].cpu().numpy() - recall).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1, 2), (255, 256, 257), (4096, 4097), (33, 0, 5000)])
def test_records_are_stored_in_stable_score_order(sizes):
    import panoptic_evaluator_gb300 as pe
    rng = np.random.default_rng(sum(sizes))
    masks, classes, scores = [], [], []
    for n in sizes:
        masks.append(torch.ones((n, 1, 16), dtype=torch.bool, device="cuda"))
        classes.append(rng.integers(0, 50, n))
        s = rng.integers(-4, 5, n) / 4.0
        s[rng.random(n) < 0.1] = -0.0
        s[rng.random(n) < 0.05] = np.inf
        s[rng.random(n) < 0.05] = np.nan
        scores.append(s)
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    target = [torch.ones((1, 1, 16), dtype=torch.bool, device="cuda") for _ in sizes]
    ev = pe.InstanceEvaluator(50, validate=False)
    ev.update(pe.InstanceBatch(masks, [dev(c) for c in classes], [dev(s) for s in scores]),
              pe.InstanceBatch(target, [torch.zeros(1, dtype=torch.int64, device="cuda") for _ in sizes]))
    state = ev.state_dict()
    order = [np.argsort(-s, kind="stable") for s in scores]  # NaN sorts last
    np.testing.assert_array_equal(state["records.scores"].cpu().numpy(),
                                  np.concatenate([s[o] for s, o in zip(scores, order)]))
    np.testing.assert_array_equal(state["records.classes"].cpu().numpy(),
                                  np.concatenate([c[o] for c, o in zip(classes, order)]))


@pytest.mark.gpu
@pytest.mark.parametrize("areas", (False, True))
@pytest.mark.parametrize("images, dets, gts, classes", [(1, 1, 1, 1), (3, 40, 9, 2), (2, 130, 70, 33), (2, 0, 5, 3)])
def test_unchecked_updates_match_from_the_pixel_counts(images, dets, gts, classes, areas):
    """Without validation areas and classes come from other kernels: the results equal the checked update's."""
    import panoptic_evaluator_gb300 as pe
    generator = torch.Generator("cuda").manual_seed(dets + gts)
    draw = lambda n: torch.rand((n, 61, 67), device="cuda", generator=generator) < 0.3  # noqa: E731
    label = lambda n: torch.randint(0, classes, (n,), device="cuda", generator=generator)  # noqa: E731
    gm = [draw(gts) for _ in range(images)]
    pm = [torch.cat((m, draw(dets)))[:dets] for m in gm]  # copies of the targets first
    args = (pe.InstanceBatch(pm, [label(dets) for _ in pm], [torch.rand(dets, device="cuda", generator=generator) for _ in pm]),
            pe.InstanceBatch(gm, [label(gts) for _ in gm],
                             crowd=[torch.rand(gts, device="cuda", generator=generator) < 0.2 for _ in gm],
                             areas=[m.flatten(1).sum(1).float() * 2 + 0.5 for m in gm] if areas else None))
    results = []
    for validate in (True, False):
        evaluator = pe.InstanceEvaluator(classes, validate=validate)
        evaluator.update(*args)
        results.append(evaluator.compute())
    for key, value in results[0].items():
        assert torch.equal(value, results[1][key]), key
