"""A checkpoint's result views: independent of one another, as many as are read."""

import copy
import pickle

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from panoptic_evaluator_gb300 import _native as N
from panoptic_evaluator_gb300 import prefix as P

ROWS, T, C = 300, 2, 5


@pytest.fixture(params=(True, False), ids=("host", "python"))
def outputs(request, monkeypatch):
    from panoptic_evaluator_gb300 import build
    build.build()
    if not request.param:
        monkeypatch.setattr(N, "_host", False)
    return _outputs()


def _outputs():
    layout, total = P._output_layout(ROWS, T, C)
    return P.PackedOutputs(torch.arange(total + 1), layout)


def _snapshots(outputs):
    return P.unpack(outputs, 0, range(1, ROWS + 1), torch.zeros(T))


def _leaves(value):
    if isinstance(value, torch.Tensor):
        yield value
    elif not isinstance(value, int):
        for v in value.values():
            yield from _leaves(v)


def test_values_are_the_rows(outputs):
    for r in (0, 1, ROWS - 1):
        s = _snapshots(outputs)[r]
        for key, field in (("tp", "tp"), ("iou_sum", "sums"), ("confusion", "confusion"), ("miou", "miou")):
            want = outputs[field][r]
            assert s[key].dtype is want.dtype and s[key].shape == want.shape and s[key].data_ptr() == want.data_ptr()
        for i, group in enumerate(("All", "Things", "Stuff")):
            for m, metric in enumerate(("pq", "sq", "rq")):
                assert s[group][metric].data_ptr() == outputs["summaries"][r, i, m].data_ptr()
                assert s[group][metric].shape == ()
            assert s[group]["n"].data_ptr() == outputs["counts"][r, i].data_ptr()
        for m, metric in enumerate(("pq", "sq", "rq", "iou")):
            assert torch.equal(s["per_class"][metric].view(torch.int64), outputs["values"].view(torch.int64)[r, m])
        for key, field in (("tp", "itp"), ("fp", "ifp"), ("fn", "ifn"), ("precision", "precision"),
                           ("recall", "recall")):
            want = outputs[field][r]
            got = s["instance"][key]
            assert got.dtype is want.dtype and got.shape == want.shape and got.data_ptr() == want.data_ptr()


def test_one_checkpoint_makes_only_its_own_views(outputs):
    made = []

    class Count(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            result = func(*args, **(kwargs or {}))
            made.append(len(result) if isinstance(result, (list, tuple)) else 1)
            return result
    last = _snapshots(outputs)[-1]
    with Count():
        for key in last:
            last[key]
    assert sum(made) <= 150


def test_every_view_can_be_changed_in_place(outputs):
    weight = torch.ones((), dtype=torch.float64, requires_grad=True)
    for k in range(len(list(_leaves(dict(_snapshots(outputs)[7]))))):
        value = list(_leaves(dict(_snapshots(_outputs())[7])))[k]
        if value.is_floating_point():
            value.mul_(weight)
            assert value.requires_grad
        else:
            value.add_(1)


def test_an_index_outside_the_field_is_refused(outputs):
    part = N.host().part if N.host() is not None else P._part
    for row, *index in ((ROWS,), (0, C), (0, 0, 0)):
        with pytest.raises(IndexError):
            part(outputs, row, "tp", *index)


def test_a_snapshot_can_be_copied_and_pickled(outputs):
    snapshot = _snapshots(outputs)[3]
    for again in (pickle.loads(pickle.dumps(snapshot)), copy.deepcopy(snapshot)):
        assert torch.equal(again["confusion"], snapshot["confusion"])
