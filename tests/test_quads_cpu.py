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
