"""When a master pattern gets a gather table, and what happens when it cannot."""

import pytest
import torch

from ebsdtorch_b200 import kernels
from ebsdtorch_b200.kernels import RowBuffers


def _master(h):
    return torch.empty((h, 2 * h), device="meta")


@pytest.mark.parametrize("h,samples,made", [(251, 1 << 22, True), (251, (1 << 22) - 1, False), (1001, 1 << 22, False),
                                            (1001, 4 * 1001 * 2002, True), (3001, 1 << 40, True),
                                            (4001, 1 << 40, False)])
def test_rule(monkeypatch, h, samples, made):
    monkeypatch.setattr(kernels, "sampling_quads", lambda mp: "table")
    assert kernels.quads_for(_master(h), samples) == ("table" if made else None)


def test_no_room_for_a_table_means_none(monkeypatch):
    def full(mp):
        raise torch.OutOfMemoryError("full")

    monkeypatch.setattr(kernels, "sampling_quads", full)
    assert kernels.quads_for(_master(1001), 1 << 30) is None


def _project(monkeypatch, quads, h=4):
    names = []
    monkeypatch.setattr(kernels, "_cuda", lambda t, name, dtype=None, contiguous=True: t)
    monkeypatch.setattr(kernels, "_stream", lambda d: None)
    monkeypatch.setattr(kernels, "call", lambda name, *a: names.append(name))
    monkeypatch.setattr(kernels, "sampling_quads", lambda mp: torch.zeros((*mp.shape, 4)))
    monkeypatch.setattr(kernels, "QUADS_MIN_SAMPLES", 1)
    kernels.project(torch.zeros(h, 2 * h), torch.zeros(3, 50), torch.zeros(10, 4), RowBuffers(), quads=quads)
    return names


def test_route_without_a_table_can_be_asked_for(monkeypatch):
    assert _project(monkeypatch, None) == ["ebsd_project_dictionary_quads"]
    assert _project(monkeypatch, False) == ["ebsd_project_dictionary"]
    assert _project(monkeypatch, torch.zeros(4, 8, 4)) == ["ebsd_project_dictionary_quads"]


@pytest.mark.parametrize("shape", [(4, 8), (4, 7, 4), (3, 8, 4), (128,)])
def test_table_of_another_image_is_refused(monkeypatch, shape):
    """The kernel indexes the table by the master pattern's sizes."""
    with pytest.raises(ValueError, match="table"):
        _project(monkeypatch, torch.zeros(shape))
