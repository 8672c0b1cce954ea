"""The host path's extension module belongs to one torch and Python; without it the Python host path serves."""

import warnings

import pytest
import torch

from panoptic_evaluator_gb300 import _native as N
from panoptic_evaluator_gb300 import build


@pytest.fixture
def built():
    build.build()


def test_another_torch_makes_the_build_stale(built, monkeypatch):
    assert not build.stale()
    monkeypatch.setattr(build, "host_tag", lambda: "another torch")
    assert build.stale()


@pytest.mark.parametrize("tag", ("another torch", None))
def test_a_module_of_another_torch_is_not_opened(tag, built, monkeypatch, tmp_path):
    path = tmp_path / "_host.tag"
    if tag:
        path.write_text(tag)
    monkeypatch.setattr(N, "HOST_TAG", path)
    monkeypatch.setattr(N, "_host", None)
    with pytest.warns(RuntimeWarning, match="built"):
        assert N.host() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert N.host() is None  # said once


def test_a_failed_compilation_is_a_warning_and_is_not_repeated(built, monkeypatch, tmp_path):
    def fails(verbose=False):
        raise RuntimeError("no headers")
    monkeypatch.setattr(build, "HOST_TAG", tmp_path / "_host.tag")
    monkeypatch.setattr(build, "HOST_MODULE", tmp_path / "_host.so")
    monkeypatch.setattr(build, "compile_host", fails)
    assert build.stale()
    with pytest.warns(RuntimeWarning, match="no headers"):
        build.build_host()
    assert not build.stale()


@pytest.mark.gpu
def test_evaluators_without_the_module(monkeypatch):
    import panoptic_evaluator_gb300 as pe
    maps = torch.zeros((1, 8, 24), dtype=torch.int32, device="cuda")
    maps[:, 4:] = 1
    classes = torch.tensor([[-1, 0]], dtype=torch.int32, device="cuda")
    crowd = torch.zeros((1, 2), dtype=torch.bool, device="cuda")
    masks, labels = [maps == 1], [torch.zeros(1, dtype=torch.int64, device="cuda")]
    target, detections = pe.PanopticBatch(maps, classes, crowd), pe.InstanceBatch(masks, labels, [labels[0].float()])

    def results():
        joint = pe.SegmentationEvaluator(1)
        for _ in range(2):
            joint.reset()
            joint.update(target, detections, target)
        prefix, = pe.segmentation_prefixes(pe.InstanceBatch(masks, labels), target, 1)
        score, = pe.panoptic_quality(target, target, 1)
        return (joint.compute()["instance"]["ap"], joint.compute()["All"]["pq"], prefix[0]["All"]["pq"], score)
    expected = [float(v) for v in results()]
    monkeypatch.setattr(N, "_host", False)
    assert [float(v) for v in results()] == expected
