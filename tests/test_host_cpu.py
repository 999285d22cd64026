"""The module that calls the library with tensors (csrc/gaac_host.cpp): the same answers as the ctypes binding to calls that the library refuses, and what its arguments may be.  Every call
here is refused before memory is touched."""
import sys
import threading
import types
import pytest
import torch
from gaac_b200 import _lib


def _t(n=64, dtype=torch.uint8): return torch.zeros(n, dtype=dtype)


def test_the_same_refusals_as_through_ctypes():
    H, L = _lib.host(), _lib.lib()
    u8, i32, ws = _t(), _t(64, torch.int32), _t(64)
    side = (u8, u8, i32, i32, u8, i32, u8, u8, None)
    page = types.SimpleNamespace(sm=u8, codes=u8, flags=i32, tile_off=i32, ovf=u8, ovf_head_start=i32, base3=u8, base4=u8)
    c_side = _lib.Side(u8.data_ptr(), u8.data_ptr(), i32.data_ptr(), i32.data_ptr(), u8.data_ptr(), i32.data_ptr(), u8.numel(), u8.data_ptr(), u8.data_ptr(), None)
    q, p = u8, u8.data_ptr()
    for S_pad, nsplit, G, off in ((16, 1, 4, 0), (17, 1, 4, 0), (16, 0, 4, 0), (16, 1, 9, 0), (16, 2000, 4, 0), (16, 1, 4, 1)):           # too small a workspace; then an argument each
        got = H.gaac_decode_attn_pages(page, side, q[off:], 1, G, 1, 16, S_pad, 0.1, nsplit, 1, ws, ws.numel(), u8, None, None, None, 0, None)
        want = L.gaac_decode_attn_pages(c_side, c_side, p + off, 1, G, 1, 16, S_pad, 0.1, nsplit, 1, ws.data_ptr(), ws.numel(), p, None, None, None, 0, None)
        assert got == want != 0, (S_pad, nsplit, G, off)
        for name in ("gaac_decode_attn", "gaac_decode_attn_balanced", "gaac_decode_attn_flat"):
            got = getattr(H, name)(side, side, p + off, i32, 1, G, 1, i32, S_pad, 0.1, nsplit, None, 0, 1, ws, ws.numel(), u8, None, None)
            want = getattr(L, name)(c_side, c_side, p + off, i32.data_ptr(), 1, G, 1, i32.data_ptr(), S_pad, 0.1, nsplit, None, 0, 1, ws.data_ptr(), ws.numel(), p, None, None)
            assert got == want != 0, (name, S_pad, nsplit, G, off)
    for TS in (3008, 3007, 2896):
        fields = (u8, u8, i32, None, None, None, u8, u8, u8, u8, 1, TS, 128)
        c_paged = _lib.Paged(p, p, i32.data_ptr(), None, None, None, p, p, p, p, 1, TS, 128)
        for name in ("gaac_paged_decode_attn", "gaac_paged_decode_attn_balanced", "gaac_paged_decode_attn_flat", "gaac_paged_decode_attn256", "gaac_paged_decode_attn256_flat"):
            got = getattr(H, name)(fields, i32, 4, i32, q, 1, 4, 0.1, 1, ws, ws.numel(), u8, None, None)
            assert got == getattr(L, name)(c_paged, i32.data_ptr(), 4, i32.data_ptr(), p, 1, 4, 0.1, 1, ws.data_ptr(), ws.numel(), p, None, None) != 0, (name, TS)
        assert H.gaac_paged_store(fields, u8, u8, 127, 128, i32, 1, i32, None) == L.gaac_paged_store(c_paged, p, p, 127, 128, i32.data_ptr(), 1, i32.data_ptr(), None) != 0
        assert H.gaac_paged_decode_blocks(fields, i32, 0, u8, u8, 128, None) == L.gaac_paged_decode_blocks(c_paged, i32.data_ptr(), 0, p, p, 128, None) != 0
    store = types.SimpleNamespace(sm=u8, codes=u8, flags=i32, tile_off=i32, ovf=u8, ovf_used=i32, tail=u8, base3=u8, base4=u8)
    c_store = _lib.Store(p, p, i32.data_ptr(), i32.data_ptr(), p, i32.data_ptr(), p, p, p)
    a = (p, p, i32.data_ptr(), -1, 1, i32.data_ptr(), i32.data_ptr(), 16, 64, 1, i32.data_ptr(), None)
    assert H.gaac_append_kv(store, store, *a) == L.gaac_append_kv(c_store, c_store, *a) != 0
    a = (p, p, -1, 128, 0, 1, i32.data_ptr(), i32.data_ptr(), 16, 64, 1, p, 64, i32.data_ptr())
    assert H.gaac_cache_prefill_own(store, store, *a, p, 64, None) == L.gaac_cache_prefill_own(c_store, c_store, *a, p, 64, None) != 0
    assert H.gaac_cache_prefill(store, store, *a, 0, None) == L.gaac_cache_prefill(c_store, c_store, *a, 0, None) != 0


def test_arguments():
    H = _lib.host()
    u8, i32 = _t(), _t(64, torch.int32)
    duck = types.SimpleNamespace(data_ptr=lambda: 0, numel=lambda: 64)
    fields = lambda **k: tuple(k.get(n, d) for n, d in (("buf", u8), ("raw", duck), ("mt", i32), ("stack", None), ("top", None), ("err", None), ("b3k", u8), ("b4k", u8), ("b3v", u8), ("b4v", u8),
                                                       ("n_kv", 1), ("TS", 3008), ("slot", 128)))
    call = lambda f, n=1: H.gaac_paged_decode_blocks(f, i32, n, u8, u8, 128, None)
    assert call(fields()) != 0                                                             # what has a data_ptr is taken; a null one is refused by the library
    with pytest.raises(TypeError): call(fields()[:12])
    with pytest.raises(TypeError): call(list(fields()))
    with pytest.raises((TypeError, AttributeError)): call(fields(raw="raw"))
    with pytest.raises(TypeError): call(fields(), 1.5)
    with pytest.raises(OverflowError): call(fields(), 1 << 40)                             # (an int of the C side)
    with pytest.raises(TypeError): H.gaac_paged_decode_blocks(fields(), i32, 1, u8, u8, 128)
    with pytest.raises(AttributeError): H.gaac_append_kv(duck, duck, *[None] * 12)         # no store


def test_empty():
    H = _lib.host()
    like = torch.zeros(2, dtype=torch.float32)
    for kind, dtype in ((0, torch.uint8), (1, torch.int32), (2, torch.bfloat16), (3, torch.float32)):
        t = H.empty(like, kind, 3, 0, 5)
        assert t.shape == (3, 0, 5) and t.dtype == dtype and t.device == like.device and t.is_contiguous() and not t.requires_grad
    with pytest.raises(RuntimeError): H.empty(like, 0, -1)
    with pytest.raises(TypeError): H.empty(None, 0, 1)
    with pytest.raises(TypeError): H.empty(like, 0, 1, 1, 1, 1, 1)


def test_other_threads_run_while_memory_is_allocated():
    """The allocator may wait for a GPU, which may wait for another thread's launch.  With a switch interval that never ends a thread runs only where this one lets go of the interpreter."""
    H, like = _lib.host(), torch.zeros(1)
    ran, started, interval = [], threading.Event(), sys.getswitchinterval()
    gate = threading.Lock()
    gate.acquire()

    def other():
        started.set()
        with gate: ran.append(1)

    t = threading.Thread(target=other)
    t.start()
    started.wait()
    sys.setswitchinterval(1000.0)
    try:
        gate.release()
        kept = []                                    # (to free one lets go of the interpreter as well)
        for _ in range(10000):
            kept.append(H.empty(like, 0, 1 << 20))
            if ran: break
        assert ran
    finally:
        sys.setswitchinterval(interval)
        t.join()
