"""Counters kept between calls: one buffer per stream for all users, no more than so many, given back with the last user."""
import gc
import weakref
import pytest
from common import to_bf16_cuda


class User:
    _kept = None


def test_buffers_of_a_stream():
    import torch
    from gaac_b200 import _lib
    kept, dev, a, b = _lib.Kept("int64"), torch.device("cpu"), User(), User()
    t = kept.of(a, dev, 7, 4)
    assert t.dtype == torch.int64 and not t.any() and kept.of(b, dev, 7, 3) is t and kept.of(a, dev, 8, 4) is not t
    wide = kept.of(b, dev, 7, 5)
    assert wide.numel() >= 5 and kept.of(a, dev, 7, 4) is wide and len(kept) == 2
    refs = [weakref.ref(x) for x in kept.values()]
    del t, wide
    for _ in range(3):
        for s in range(100):
            assert not kept.of(a, dev, s, 1).any() and len(kept) <= kept.MOST
    assert kept.of(a, dev, 99, 1) is kept.of(b, dev, 99, 1)
    del a
    gc.collect()
    assert len(kept) == kept.MOST                    # b is there
    del b
    gc.collect()
    assert len(kept) == 0 and kept.values() == [] and all(r() is None for r in refs)
    c = User()
    assert kept.of(c, dev, 7, 1).numel() == 1 and len(kept) == 1


def test_copies_and_pickles_of_a_user():
    import copy
    import pickle
    import torch
    from gaac_b200 import Codec, _lib
    kept, codec, dev = _lib.ENCODE_COUNTERS, Codec(1, "cpu"), torch.device("cpu")
    t = kept.of(codec, dev, 7, 1)
    for other in (copy.copy(codec), copy.deepcopy(codec), pickle.loads(pickle.dumps(codec))):
        assert kept.of(other, dev, 7, 1) is t
    assert pickle.loads(pickle.dumps(codec)).__dict__["_kept"] is None          # nothing of the GPU's is written


def test_many_threads():
    import threading
    import torch
    from gaac_b200 import _lib
    kept, dev, users, errors = _lib.Kept("uint8"), torch.device("cpu"), [User() for _ in range(4)], []

    def work(i):
        try:
            for n in range(3000):
                assert kept.of(users[i], dev, n % 40, 1 + n % 5).numel() >= 1 + n % 5
                if n % 100 == 0: users[i] = User()
        except BaseException as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads: t.start()
    for t in threads: t.join()
    assert not errors and len(kept) <= kept.MOST


@pytest.mark.gpu
def test_what_the_calls_keep():
    """A cache and a codec on 70 streams: what they keep is bounded, and gone with them."""
    import torch
    import numpy as np
    from gaac_b200 import Codec, CompressedKVCache, encoder, kv_cache
    from oracle import gaac_oracle as O
    x = to_bf16_cuda(O.kv_like(2, 100, seed=1))
    rows = x.transpose(0, 1).contiguous()
    cache, codec = CompressedKVCache(1, 2, 112), Codec(2).calibrate(x)
    ref = codec.encode(x, "k")
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(40)]
    torch.cuda.synchronize()
    for s in streams + streams[:3]:
        with torch.cuda.stream(s):
            cache.prefill(0, rows, rows)
            page = codec.encode(x, "k")
            assert torch.equal(page.ovf, ref.ovf) and torch.equal(cache.decompress(0)[0].view(torch.int16), rows.view(torch.int16))
        torch.cuda.synchronize()
    assert len({s.cuda_stream for s in streams}) > 40
    for kept in (kv_cache._TABLES, encoder._COUNTERS):
        assert 1 <= len(kept) <= 32 and not any(bool(t.any()) for t in kept.values())
    del cache, codec
    gc.collect()
    assert len(kv_cache._TABLES) == 0 and len(encoder._COUNTERS) == 0
