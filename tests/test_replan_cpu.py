"""A plan made from the allocator's cache is made again from the driver's free
memory when the allocator cannot serve it (fragments, blocks of CUDA graphs'
pools); a plan that had asked the driver, or that the caller bounded, is not."""

import pytest
import torch

from ebsdtorch_b200 import engine
from ebsdtorch_b200.engine import SearchConfig, Searcher
from ebsdtorch_b200.kernels import TILE_D, TILE_Q, round_up

N_DICT, N_Q, N_PIX = 36829, 4096, 3600


class _Served(Exception):
    pass


def _run(monkeypatch, cached, free, limit, **cfg):
    """The row counts that a search asks the allocator for when no block above
    `limit` rows can be had, until both row sets are there."""
    monkeypatch.setattr(engine, "cached_bytes", lambda d: cached)
    monkeypatch.setattr(engine, "default_budget", lambda d: int(0.9 * free))
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: asked.append("empty"))
    asked, held = [], []

    def rows(n_rows, n_pix, pad_rows, *a, **k):
        asked.append(n_rows)
        if n_rows > limit:
            raise torch.OutOfMemoryError("no block of this size")
        held.append(n_rows)
        if pad_rows == TILE_Q:
            raise _Served

    monkeypatch.setattr(engine, "RowSet", type("Rows", (engine.RowSet,), {"__new__": lambda c, *a, **k: rows(*a, **k)}))
    s = Searcher(N_DICT, N_Q, N_PIX, 1, SearchConfig(**cfg), "cuda:0")
    s.device = torch.device("cpu")  # the outputs of run() are allocated there
    try:
        s.run(None, None)
    except _Served:
        pass
    return asked, s


def test_plan_from_the_cache_falls_back_to_the_driver(monkeypatch):
    asked, s = _run(monkeypatch, 1 << 40, 300 << 20, 20000)
    assert asked[0] == round_up(N_DICT, TILE_D)  # everything at once
    assert asked[1] == "empty"  # what the first attempt held goes back before the driver is asked
    assert asked[2] < 20000 and asked[2] == s.dict_chunk and asked[3] == s.query_chunk


@pytest.mark.parametrize("cached,cfg", [(0, {}), (1 << 40, {"workspace_bytes": 10 << 30})])
def test_other_plans_raise(monkeypatch, cached, cfg):
    with pytest.raises(torch.OutOfMemoryError):
        _run(monkeypatch, cached, 10 << 30, 20000, **cfg)


def test_second_failure_raises(monkeypatch):
    with pytest.raises(torch.OutOfMemoryError):
        _run(monkeypatch, 1 << 40, 10 << 30, 20000)
