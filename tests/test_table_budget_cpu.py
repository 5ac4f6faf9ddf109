"""The projector's gather table under a budget that the caller gives: rows and
table together stay within it, and where the table has no room the plan is the
one without it."""

import pytest
import torch

from ebsdtorch_b200 import kernels
from ebsdtorch_b200.ebsd import indexing
from ebsdtorch_b200.engine import RowSet, SearchConfig, Searcher
from ebsdtorch_b200.kernels import DT_BF16

N_DICT, N_Q, N_PIX = 100000, 5000, 3600
TABLE = 16 * 1001 * 2002


def _plan(monkeypatch, budget):
    made = []
    monkeypatch.setattr(kernels, "sampling_quads", lambda mp: made.append(1) or "table")
    cfg = SearchConfig(workspace_bytes=budget)
    s, table = indexing._plan_search(torch.empty((1001, 2002), device="meta"), N_DICT * N_PIX, N_DICT, N_Q, N_PIX, 1,
                                     cfg, "cpu")
    assert not made  # not before the rows have their memory
    tables = table(), table()
    assert tables[0] is tables[1] and len(made) == (tables[0] == "table")
    row = RowSet.bytes_per_row(N_PIX, DT_BF16, True)
    return tables[0], s, s.dict_chunk * row + s.query_chunk * (row + 12), Searcher(N_DICT, N_Q, N_PIX, 1, cfg, "cpu")


@pytest.mark.parametrize("budget", [8 * TABLE, 1 << 30, 4 << 30])
def test_table_comes_out_of_the_budget(monkeypatch, budget):
    table, _, planned, _ = _plan(monkeypatch, budget)
    assert table == "table" and planned + TABLE <= budget


@pytest.mark.parametrize("budget", [20 << 20, 8 * TABLE - 1])
def test_small_budgets_go_to_the_rows(monkeypatch, budget):
    table, s, planned, without = _plan(monkeypatch, budget)
    assert table is False and planned <= budget
    assert (s.dict_chunk, s.query_chunk) == (without.dict_chunk, without.query_chunk)


def test_too_small_for_anything_is_refused(monkeypatch):
    with pytest.raises(MemoryError):
        _plan(monkeypatch, 1 << 20)
