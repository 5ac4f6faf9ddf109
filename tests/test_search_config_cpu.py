"""SearchConfig's fields keep their positions: a new one goes to the end."""

from ebsdtorch_b200.engine import SearchConfig


def test_positional_fields():
    cfg = SearchConfig("fp8", 16, "cosine", 1 << 30, 4096, 2048, 1024, 128, 2, 3, True, False)
    assert (cfg.query_chunk, cfg.dict_chunk, cfg.max_query_chunk) == (4096, 2048, 1024)
    assert (cfg.tile_n, cfg.splits, cfg.wave_tiles, cfg.persistent, cfg.rescore_gate) == (128, 2, 3, True, False)
    assert cfg.free_share == 1.0
