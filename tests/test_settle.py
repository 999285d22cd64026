"""The host check of prefills made with check=False: which status words it reads, and that the number of slots is not what it costs."""
import time
import pytest


def _cache(n_slots):
    import torch
    import gaac_b200.kv_cache as kvc
    cache = object.__new__(kvc.CompressedKVCache)
    cache.n_slots, cache.S, cache._pending_bytes = n_slots, torch.zeros(1), 0
    cache._slot_status = torch.zeros(n_slots, 4, dtype=torch.int32)
    cache.k = type("Store", (), {"ovf_cap": 1 << 20})()
    cache.repaired = []
    cache._prefill_launch = lambda slot, L, k, v, scratch, status, copy_only: cache.repaired.append((slot, L, status.tolist()))
    cache._grow = lambda need: cache.repaired.append(("grow", need))
    return cache


@pytest.mark.parametrize("n_slots", [1, 7, 64, 65, 4096, 4097, 8192, 8193])
def test_words_of_the_pending_slots_are_read(n_slots):
    import torch
    from gaac_b200.kv_cache import TILE_MAX_ESC, _OVER_READ
    cache = _cache(n_slots)
    slots = sorted({0, n_slots // 2, n_slots - 1}, reverse=True)
    for i, s in enumerate(slots):
        cache._slot_status[s] = torch.tensor([i, 100 + i, 0, (1 << 20) + i])                # the first one fits, the others are copied again
    cache._pending = {s: (10 + i, None) for i, s in enumerate(slots)}
    cache.settle_prefills()
    want = [("grow", (1 << 20) + len(slots) - 1 + TILE_MAX_ESC + _OVER_READ)] + [(s, 10 + i, [i, 100 + i, 0, (1 << 20) + i]) for i, s in enumerate(slots) if i]
    assert cache.repaired == want and not cache._pending


def test_many_slots_cost_little_more_than_few():
    best = {}
    for n_slots in (4, 4096):
        cache, best[n_slots] = _cache(n_slots), 1.0
        for _ in range(50):
            cache._pending = {0: (16, None), 3: (16, None)}
            t = time.perf_counter()
            cache.settle_prefills()
            best[n_slots] = min(best[n_slots], time.perf_counter() - t)
    assert best[4096] < 20 * best[4], best            # (about the same; with every slot's words made into Python numbers more than 100 times as much)
