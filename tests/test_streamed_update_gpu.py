"""Instance updates whose masks are streamed, at the sizes of one image and less, through the launches an update makes.

Such batches are small enough to be contracted whatever their masks hold, so the rule that decides by size is replaced;
the scratch holds what an earlier call may have left. FP64 results agree with the oracle within 1e-12.
"""

import ctypes

import numpy as np
import pytest
import torch

from helpers import assert_tree, cuda
from panoptic_evaluator_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture
def always_streamed():
    host = N.host()
    addresses = {name: ctypes.cast(getattr(N.library(), name), ctypes.c_void_p).value for name in N.SIGNATURES}
    rule = ctypes.CFUNCTYPE(ctypes.c_int64, *[ctypes.c_void_p] * 4, ctypes.c_int64, ctypes.c_int64)(
        lambda *_: calls.append(2**62) or calls[-1])
    calls = []
    host.bind({**addresses, "pe_stream_limit": ctypes.cast(rule, ctypes.c_void_p).value})
    yield calls
    host.bind(addresses)


@pytest.mark.parametrize("validate", (False, True))
@pytest.mark.parametrize("images", [
    [(1, 1, 1, 1)], [(3, 2, 5, 7)], [(5, 0, 33, 31), (0, 4, 20, 9), (0, 0, 4, 4), (2, 2, 16, 16)],
    [(17, 63, 64, 64)], [(33, 64, 63, 65)], [(130, 130, 61, 67)], [(300, 5, 40, 40)],
    [(6, 33, 127, 33), (7, 9, 64, 512), (100, 8, 37, 111)], [(20, 12, 4096, 1), (20, 12, 4097, 1), (20, 12, 4095, 1)],
    [(40, 20, 700, 500)], [(9, 7, 30 + 3 * k, 41) for k in range(40)],
])
def test_small_streamed_updates(images, validate, always_streamed):
    import panoptic_evaluator_gb300 as pe
    from oracle import instance as oinst
    rng = np.random.default_rng(len(images) + images[0][0])
    pm, gm, pc, gc, scores, crowd = [], [], [], [], [], []
    for d, g, h, w in images:
        masks = rng.random((d + g, h * w)) < 0.02
        masks[np.arange(d + g), rng.integers(0, h * w, d + g)] = True
        copies = rng.integers(0, max(g, 1), d)  # half of the detections: a target with some pixels more
        if g:
            masks[:d:2] |= masks[d + copies[::2]]
        pm.append(masks[:d].reshape(d, h, w))
        gm.append(masks[d:].reshape(g, h, w))
        gc.append(rng.integers(0, 3, g))
        pc.append(np.where(np.arange(d) % 2 == 0, gc[-1][copies] if g else 0, rng.integers(0, 3, d)))
        scores.append(rng.random(d))
        crowd.append(rng.random(g) < 0.1)
    oracle = oinst.InstanceOracle(3)
    oracle.update(pm, pc, scores, gm, gc, crowd)
    ev = pe.InstanceEvaluator(3, validate=validate)
    ev._arena = torch.full((32 << 20,), 0xa5, dtype=torch.uint8, device="cuda")
    arena = ev._arena
    ev.update(pe.InstanceBatch([cuda(m) for m in pm], [cuda(c) for c in pc], [cuda(s) for s in scores]),
              pe.InstanceBatch([cuda(m) for m in gm], [cuda(c) for c in gc], crowd=[cuda(c) for c in crowd]))
    assert ev._arena is arena and always_streamed  # the update took the host path, this scratch and the rule
    assert_tree(ev.compute(), oracle.compute())
