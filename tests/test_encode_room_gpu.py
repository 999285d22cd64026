"""Codec.encode around the room that it makes for the escape bytes before it knows their number: exactly enough, a byte less, far less, none; and an allocation that fails
while the kernels run."""
import numpy as np
import pytest
from common import to_bf16_cuda, page_to_dict, assert_pages_equal
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["k", "v"])
def test_room(kind, monkeypatch):
    import torch
    from gaac_b200 import Codec, encoder
    x16, n_kv = O.kv_like(3, 333, seed=2), 3
    x = to_bf16_cuda(x16)
    c = Codec(n_kv).calibrate(x)
    ref = O.encode(x16, c.base3.cpu().numpy(), c.base4.cpu().numpy(), kind, n_kv)
    n, items = int(ref["ovf_head_start"][-1]), 3 * 21
    for room in (n / items, (n - 1) / items, (n + 1) / items, 8, 0, 1280):
        class Exact(float):                          # items * ROOM is the whole number that is meant
            def __rmul__(self, other): return int(round(float(self) * other))
        monkeypatch.setattr(encoder, "ROOM", Exact(room))
        for _ in range(2):
            pg = c.encode(x, kind)
            assert pg.ovf.numel() == n + 8 and bool((pg.ovf[n:] == 0).all())
            assert_pages_equal(page_to_dict(pg), ref)
            assert torch.equal(Codec.decode(pg).view(torch.int16), x.view(torch.int16))
            assert len(encoder._COUNTERS) >= 1 and not any(int(w) for w in encoder._COUNTERS.values())


def test_failed_allocation_waits_for_the_kernels(monkeypatch):
    import torch
    from gaac_b200 import Codec, _lib
    x16 = O.kv_like(2, 100, seed=2)
    x = to_bf16_cuda(x16)
    c = Codec(2).calibrate(x)
    lib, waits, empty = _lib.lib(), [], torch.empty

    class Counting:
        def __getattr__(self, name):
            if name == "gaac_wait_total": waits.append(1)
            return getattr(lib, name)

    def failing(*shape, **kw):
        if shape == (2, 100): raise torch.OutOfMemoryError("no room")
        return empty(*shape, **kw)
    with monkeypatch.context() as m:
        m.setattr(_lib, "lib", lambda: Counting())
        m.setattr(torch, "empty", failing)
        with pytest.raises(torch.OutOfMemoryError):
            c.encode(x, "k")
    assert len(waits) == 1
    assert_pages_equal(page_to_dict(c.encode(x, "k")), O.encode(x16, c.base3.cpu().numpy(), c.base4.cpu().numpy(), "k", 2))


def test_refused_in_a_capture():
    """A counter made in a capture would be zero only when the graph runs: the encode is refused, and works on that stream afterwards."""
    import torch
    from gaac_b200 import Codec
    x16 = O.kv_like(2, 100, seed=2)
    x = to_bf16_cuda(x16)
    c = Codec(2).calibrate(x)
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(g, stream=side):
            c.encode(x, "k")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        pg = c.encode(x, "k")
    torch.cuda.synchronize()
    assert_pages_equal(page_to_dict(pg), O.encode(x16, c.base3.cpu().numpy(), c.base4.cpu().numpy(), "k", 2))


@pytest.mark.parametrize("H,n_kv", [(3, 3), (96, 3)])                           # prefix over the heads by one warp; by a whole CTA
def test_sized_entry_point(H, n_kv):
    """gaac_encode_sized, for C callers: the total, the offsets and the tiles of Codec.encode."""
    import torch
    from gaac_b200 import Codec, _lib
    x16 = np.ascontiguousarray(np.resize(O.kv_like(n_kv, 333, seed=2), (H, 333, 128)))
    x, S, nt = to_bf16_cuda(x16), 333, 21
    c = Codec(n_kv).calibrate(x)
    page, lib = c.encode(x, "v"), _lib.lib()
    u8, i32 = dict(dtype=torch.uint8, device="cuda"), dict(dtype=torch.int32, device="cuda")
    sm, codes, slots = torch.empty(H, nt * 2048, **u8), torch.empty(H, nt * 768, **u8), torch.empty(H * nt * 1280, **u8)
    flags, sizes, off, sums, ends = torch.empty(H, nt * 16, **i32), torch.empty(H * nt, **i32), torch.empty(H, nt, **i32), torch.empty(H, **i32), torch.empty(H + 1, **i32)
    total = torch.full((1,), -1, dtype=torch.int32, pin_memory=True)
    _lib.check(lib.gaac_encode_sized(x.data_ptr(), H, S, S, nt * 16, c.base3.data_ptr(), c.base4.data_ptr(), None, n_kv, 1, sm.data_ptr(), codes.data_ptr(), flags.data_ptr(), slots.data_ptr(),
                                     sizes.data_ptr(), off.data_ptr(), sums.data_ptr(), ends.data_ptr(), total.data_ptr(), _lib.stream_ptr(x.device)), "gaac_encode_sized")
    assert int(total) == int(page.ovf_head_start[-1])                           # (it has waited: the word is read before anything else)
    for got, ref in ((sm, page.sm), (codes, page.codes), (flags, page.flags), (off, page.tile_off), (ends, page.ovf_head_start)):
        assert torch.equal(got, ref)
