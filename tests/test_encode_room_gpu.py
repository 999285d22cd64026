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
