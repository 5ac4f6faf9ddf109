"""The budget of a search: the allocator's cache when all rows fit it, else
the driver's free memory, scaled by the caller's share; the same plan either
way whenever everything fits."""

import pytest

from ebsdtorch_b200 import engine
from ebsdtorch_b200.engine import RowSet, SearchConfig, Searcher
from ebsdtorch_b200.kernels import DT_BF16, TILE_D, TILE_Q, round_up


def _searcher(monkeypatch, cached, free, n_dict, n_q, n_pix, **cfg):
    asked = []
    monkeypatch.setattr(engine, "cached_bytes", lambda d: cached)
    monkeypatch.setattr(engine, "default_budget", lambda d: asked.append(d) or int(0.9 * free))
    return Searcher(n_dict, n_q, n_pix, 1, SearchConfig(**cfg), "cuda:0"), asked


@pytest.mark.parametrize("n_dict,n_q,n_pix", [(1, 1, 1), (579, 64, 576), (36829, 4096, 3600), (36829, 4097, 3601)])
@pytest.mark.parametrize("share", [1.0, 0.7])
def test_cached_plan_is_the_whole_problem(monkeypatch, n_dict, n_q, n_pix, share):
    row = RowSet.bytes_per_row(n_pix, DT_BF16, True)
    whole = round_up(n_dict, TILE_D) * row + round_up(n_q, TILE_Q) * (row + 12)
    s, asked = _searcher(monkeypatch, int(whole / (0.9 * share)) + 2, 1 << 40, n_dict, n_q, n_pix, free_share=share)
    t, asked_t = _searcher(monkeypatch, 0, 1 << 40, n_dict, n_q, n_pix, free_share=share)
    assert not asked and asked_t
    assert (s.dict_chunk, s.query_chunk) == (t.dict_chunk, t.query_chunk)
    assert s.dict_chunk == round_up(n_dict, TILE_D) and s.query_chunk == round_up(n_q, TILE_Q)


def test_short_cache_asks_the_driver(monkeypatch):
    s, asked = _searcher(monkeypatch, 1 << 20, 200 << 20, 36829, 4096, 3600)
    assert asked and s.dict_chunk < 36829
    _, asked = _searcher(monkeypatch, 1 << 40, 1 << 40, 36829, 4096, 3600, workspace_bytes=300 << 20)
    assert not asked
    with pytest.raises(MemoryError):
        _searcher(monkeypatch, 0, 1 << 16, 36829, 4096, 3600)
