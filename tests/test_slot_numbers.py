"""CompressedKVCache.prefill with the slot number as programs have it: an int, an element of an array, a tensor of one element."""
import ctypes
import types
import numpy as np
import pytest


def _cache(monkeypatch, n_slots, own):
    """A cache whose native module records what it is handed (through the argument types of the real one)."""
    import torch
    import gaac_b200.kv_cache as kvc
    from gaac_b200 import _lib
    calls = []

    class Sizes:
        def __getattr__(self, name):
            assert name.endswith("_bytes")
            return lambda *a: 4096

    class Recording:
        """The native module up to the library: what it is not handed as a number, an address or a store it would refuse."""
        def empty(self, like, kind, *sizes): return torch.empty(sizes, dtype=torch.uint8)

        def __getattr__(self, name):
            res, args = _lib._SIGNATURES[name]

            def call(*a):
                assert len(a) == len(args)
                for value, kind in zip(a, args):
                    if kind in (ctypes.POINTER(_lib.Store),):
                        assert all(hasattr(value, f) for f in ("sm", "codes", "flags", "tile_off", "ovf", "ovf_used", "tail", "base3", "base4"))
                    else: kind.from_param(value)
                calls.append((name, a))
                return 0
            return call
    monkeypatch.setattr(kvc._lib, "lib", Sizes)
    monkeypatch.setattr(kvc._lib, "host", Recording)
    monkeypatch.setattr(kvc._lib, "stream_ptr", lambda dev: 0)
    monkeypatch.setattr(kvc._lib, "capturing", lambda: False)
    cache = object.__new__(kvc.CompressedKVCache)
    cache.n_slots, cache.n_kv, cache.cap, cache.per_sequence_bases = n_slots, 2, 64, own
    cache.S = cache.tail_len = torch.zeros(2 * n_slots, dtype=torch.int32)
    cache._slot_status, cache._pending, cache._pending_bytes, cache._scratch = torch.zeros(n_slots, 4, dtype=torch.int32), {}, 0, None
    cache.pending_scratch_limit = 1 << 30
    table = torch.zeros(2 * n_slots if own else 2, 128, dtype=torch.uint8)
    cache.k = cache.v = types.SimpleNamespace(ovf_cap=1 << 20, base3=table, base4=table, **{f: table for f in ("sm", "codes", "flags", "tile_off", "ovf", "ovf_used", "tail")})
    cache._token_rows = lambda x: x
    return cache, calls


@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("form", [int, np.int64, np.int32, np.uint8, "tensor"])
def test_every_form_of_a_slot_number(monkeypatch, form, own):
    import torch
    cache, calls = _cache(monkeypatch, 5, own)
    rows = torch.zeros(20, 2, 128, dtype=torch.bfloat16)
    for slot in (0, 3, 4):
        for check in (True, False):
            cache.prefill(torch.tensor(slot) if form == "tensor" else form(slot), rows, rows, check=check)
            name, args = calls[-1]
            assert name == ("gaac_cache_prefill_own" if own else "gaac_cache_prefill") and args[6] == slot
            assert args[15] == cache._slot_status.data_ptr() + 16 * slot
            assert list(cache._pending) == ([] if check else [slot])


@pytest.mark.parametrize("slot", [1.0, "1", None, -1, 5])
def test_what_is_no_slot_is_refused(monkeypatch, slot):
    import torch
    cache, calls = _cache(monkeypatch, 5, True)
    rows = torch.zeros(20, 2, 128, dtype=torch.bfloat16)
    with pytest.raises((TypeError, AssertionError)):
        cache.prefill(slot, rows, rows)
    assert not calls
