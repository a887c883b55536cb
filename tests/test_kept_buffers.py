"""The store of buffers derived from a neighbour table (ops._InverseCache), without a GPU."""
import torch


def _cache(capacity=2):
    from clusten import ops
    return ops._InverseCache(capacity)


def test_a_written_table_is_not_found():
    cache, idx = _cache(), torch.zeros(1, 8, 8, dtype=torch.int64)
    cache.put(idx, 8, "buffer")
    assert cache.get(idx, 8) == "buffer" and cache.get(idx, 9) is None
    idx[0, 0, 0] = 1
    assert cache.get(idx, 8) is None


def test_inference_tensors_are_neither_kept_nor_looked_up():
    """They have no version counter, so a write would go unnoticed."""
    cache = _cache()
    with torch.inference_mode():
        idx = torch.zeros(1, 8, 8, dtype=torch.int64)
        assert cache.get(idx, 8) is None
        cache.put(idx, 8, "buffer")
        assert cache.get(idx, 8) is None and not cache.entries


def test_nothing_is_kept_or_looked_up_while_a_stream_captures(monkeypatch):
    """A captured build has not run, and a replay sees other indices."""
    from clusten import ops
    cache, idx = _cache(), torch.zeros(1, 8, 8, dtype=torch.int64)
    cache.put(idx, 8, "buffer")
    monkeypatch.setattr(ops, "_capturing", lambda t: True)
    assert cache.get(idx, 8) is None
    cache.put(idx, 9, "captured")
    monkeypatch.setattr(ops, "_capturing", lambda t: False)
    assert cache.get(idx, 8) == "buffer" and cache.get(idx, 9) is None
