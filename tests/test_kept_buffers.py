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


def test_a_buffer_belongs_to_the_stream_that_built_it(monkeypatch):
    """Nothing orders another stream behind the build, nor the buffer's memory behind that stream's reads."""
    from clusten import ops
    cache, idx = _cache(), torch.zeros(1, 8, 8, dtype=torch.int64)
    stream = [1]
    monkeypatch.setattr(ops, "_stream_of", lambda t: stream[0])
    cache.put(idx, 8, "first")
    stream[0] = 2
    assert cache.get(idx, 8) is None
    cache.put(idx, 8, "second")
    assert cache.get(idx, 8) == "second"
    stream[0] = 1
    assert cache.get(idx, 8) == "first"


def test_threads_share_a_store():
    """An entry found by one thread may be dropped by another before it is moved to the end."""
    import sys
    import threading
    cache = _cache(1)
    tables = [torch.zeros(1, 8, 8, dtype=torch.int64) for _ in range(4)]
    failed, stop = [], threading.Event()

    def work(k):
        try:
            while not stop.is_set():
                if cache.get(tables[k], 8) is None:
                    cache.put(tables[k], 8, k)
                if k == 0:
                    cache.clear()
        except Exception as e:  # noqa: BLE001
            failed.append(e)
            stop.set()

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        [t.start() for t in threads]
        stop.wait(2)
        stop.set()
        [t.join() for t in threads]
    finally:
        sys.setswitchinterval(interval)
    assert not failed, failed


def test_tables_beyond_the_inverse_by_groups(lib):
    """They take the way of an explicit inverse (and nothing is kept for another one)."""
    applies = lib.clusten_inverse_grouped_applies
    assert applies(9216, 48, 9216) and applies(196, 48, 196) and applies(3136, 64, 3136) and applies(16, 8, 16)
    assert not applies(12800, 48, 12800) and not applies(9, 48, 9) and not applies(8191, 64, 8191) and not applies(196, 65, 196)
