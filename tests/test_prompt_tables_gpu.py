"""A prompt's exponent tables (gaac_cache_calibrate): lengths around what 16-bit counts hold, all values alike (a counter at its largest), rows that are no whole
number of words, scratch on a 4-byte boundary; against the tables of the same rows by the oracle."""
import numpy as np
import pytest
from common import to_bf16_cuda
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


def _tables(x, L, stride, n_kv, scratch_at=0):
    import torch
    from gaac_b200 import CompressedKVCache, _lib
    lib, cache = _lib.lib(), CompressedKVCache(2, n_kv, 64)
    scratch = torch.full((lib.gaac_cache_calibrate_scratch_bytes(n_kv) + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    n = lib.gaac_cache_calibrate_scratch_bytes(n_kv)
    _lib.check(lib.gaac_cache_calibrate(cache.k.c_store(), cache.v.c_store(), x[0].data_ptr(), x[1].data_ptr(), L, stride, 1, n_kv, cache.k.base3.shape[0],
                                        scratch.data_ptr() + scratch_at, n, torch.cuda.current_stream().cuda_stream), "gaac_cache_calibrate")
    assert bool((scratch[scratch_at + n:] == 0xA5).all()) and bool((scratch[:scratch_at] == 0xA5).all())
    for st in (cache.k, cache.v):
        assert int(st.base3[:n_kv].max()) == 0 and int(st.base4[:n_kv].max()) == 0          # the other slot's rows
    return [(st.base3[n_kv:].cpu().numpy(), st.base4[n_kv:].cpu().numpy()) for st in (cache.k, cache.v)]


def _check(rows, got, n_kv):
    for x16, (b3, b4) in zip(rows, got):
        r3, r4 = O.calibrate(np.ascontiguousarray(x16.reshape(-1, n_kv, 128).transpose(1, 0, 2)), n_kv)
        assert np.array_equal(b3, r3) and np.array_equal(b4, r4)


@pytest.mark.parametrize("L", [1, 15, 127, 128, 129, 4001, 65535, 65536])
@pytest.mark.parametrize("alike", [False, True])
def test_lengths(L, alike):
    n_kv = 1 if L > 5000 else 3
    rows = [np.full((L, n_kv * 128), 0x3F80, np.uint16) if alike else np.ascontiguousarray(O.kv_like(n_kv, L, seed=s).transpose(1, 0, 2)).reshape(L, -1) for s in (1, 2)]
    _check(rows, _tables([to_bf16_cuda(r) for r in rows], L, n_kv * 128, n_kv), n_kv)


@pytest.mark.parametrize("pad,offset", [(0, 0), (1, 0), (2, 0), (3, 1), (8, 1)])
@pytest.mark.parametrize("scratch_at", [0, 4, 8, 16])
def test_strides_and_alignment(pad, offset, scratch_at):
    n_kv, L = 2, 300
    stride = n_kv * 128 + pad
    rows = [np.ascontiguousarray(O.kv_like(n_kv, L, seed=s).transpose(1, 0, 2)).reshape(L, -1) for s in (1, 2)]
    dev = []
    for r in rows:
        wide = np.zeros(L * stride + offset, np.uint16)
        wide[offset:].reshape(L, stride)[:, :n_kv * 128] = r
        dev.append(to_bf16_cuda(wide)[offset:])
    _check(rows, _tables(dev, L, stride, n_kv, scratch_at), n_kv)


@pytest.mark.parametrize("n_ch,offset", [(1, 0), (127, 0), (130, 0), (256, 1)])
def test_histogram_of_odd_channels(n_ch, offset):
    import torch
    from gaac_b200 import _lib
    x16 = O.kv_like(1, 300 * n_ch // 128 + 1, seed=4).reshape(-1)[:300 * n_ch].copy()
    x = to_bf16_cuda(np.concatenate([np.zeros(offset, np.uint16), x16]))[offset:]
    hist = torch.zeros(n_ch, 256, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib().gaac_exponent_hist(x.data_ptr(), 300, n_ch, hist.data_ptr(), torch.cuda.current_stream().cuda_stream), "gaac_exponent_hist")
    e = (x16.reshape(300, n_ch) >> 7) & 0xFF
    assert np.array_equal(hist.cpu().numpy(), np.stack([np.bincount(e[:, c], minlength=256) for c in range(n_ch)]))


@pytest.mark.parametrize("L", [1, 15, 16, 128, 129, 700, 65535, 65536])
def test_prefill_makes_the_same_tables(L):
    """gaac_cache_prefill_own: the tables of the two-call form, its counters zero again behind every call, one set of counters for caches of different sizes."""
    import torch
    from gaac_b200 import CompressedKVCache, kv_cache
    for n_kv in ((1,) if L > 1000 else (3, 1, 5)):
        rows = [np.ascontiguousarray(O.kv_like(n_kv, L, seed=10 * n_kv + s).transpose(1, 0, 2)) for s in (1, 2)]
        cache = CompressedKVCache(2, n_kv, L)
        for _ in range(2):
            cache.prefill(1, *(to_bf16_cuda(r) for r in rows))
        _check([r.reshape(L, -1) for r in rows], [(s.base3[n_kv:].cpu().numpy(), s.base4[n_kv:].cpu().numpy()) for s in (cache.k, cache.v)], n_kv)
        assert all(not bool(ws.any()) for ws in kv_cache._TABLES.values()) and len(kv_cache._TABLES) >= 1
        k, v = cache.decompress(1)
        for got, r in zip((k, v), rows):
            assert np.array_equal(got.contiguous().view(torch.int16).cpu().numpy().view(np.uint16), r)


def test_prefill_in_a_captured_graph():
    import torch
    from gaac_b200 import CompressedKVCache
    n_kv, L = 2, 300
    x = [to_bf16_cuda(np.ascontiguousarray(O.kv_like(n_kv, L, seed=s).transpose(1, 0, 2))) for s in (1, 2, 3, 4)]
    cache, k, v = CompressedKVCache(1, n_kv, L), x[0].clone(), x[1].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cache.prefill(0, k, v, check=False)
    k.copy_(x[2]); v.copy_(x[3])
    graph.replay()
    assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(cache.decompress(0), (k, v)))
    cache.prefill(0, x[0], x[1])
    assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(cache.decompress(0), x))


# one tile per warp of the encoder, from 369 tiles on two, from 553 three, from 737 four: blocks of 16, 16, 12 and 16 tiles behind it
@pytest.mark.parametrize("tiles", [0, 1, 15, 16, 17, 63, 65, 368, 369, 370, 552, 553, 555, 564, 565, 736, 737, 740])
@pytest.mark.parametrize("room", [1280, 100])                                # 100: the streams are too small, the copy is repeated into larger ones
def test_streams_behind_the_encode(tiles, room):
    """A slot's offsets, escape bytes, counters and tails against a Page of the same tokens: blocks of ordinary tiles, of tiles with every group raw, and of both."""
    import torch
    from gaac_b200 import Codec, CompressedKVCache
    n_kv, L = 8, 16 * tiles + 7
    base = O.kv_like(n_kv, max(L, 16), seed=5)
    if tiles > 64:
        wild = np.random.default_rng(2).integers(0, 65536, base.shape).astype(np.uint16)
        t = np.arange(base.shape[1]) // 16
        base = np.where(((t % 9 == 4) | ((t >= 64) & (t < 72)) | (t == tiles - 1))[None, :, None], wild, base)
    x = to_bf16_cuda(np.ascontiguousarray(base[:, :L].transpose(1, 0, 2)))
    c = Codec(n_kv).calibrate(to_bf16_cuda(O.kv_like(n_kv, 512, seed=1)))
    cache = CompressedKVCache(3, n_kv, L, bases={"k3": c.base3, "k4": c.base4, "v3": c.base3, "v4": c.base4}, ovf_bytes_per_tile=room)
    small = cache.k.ovf_cap
    for check in (True, False):
        cache.prefill(1, x, x.flip(1).contiguous(), check=check)
        cache.settle_prefills()
    heads = slice(n_kv, 2 * n_kv)
    for st, rows in ((cache.k, x), (cache.v, x.flip(1))):
        assert torch.equal(st.tail[heads, :L % 16].view(torch.int16), rows[L // 16 * 16:].transpose(0, 1).contiguous().view(torch.int16))
        if tiles == 0:
            assert int(st.ovf_used[heads].max()) == 0
            continue
        page = c.encode(rows[:16 * tiles].transpose(0, 1).contiguous(), st.kind)
        size = page.ovf_head_start[1:] - page.ovf_head_start[:-1]
        assert torch.equal(st.ovf_used[heads], size) and torch.equal(st.tile_off[heads, :tiles], page.tile_off)
        assert torch.equal(st.flags[heads, :16 * tiles], page.flags)
        at = page.ovf_head_start.tolist()
        for h in range(n_kv):
            n = at[h + 1] - at[h]
            o = (n_kv + h) * st.ovf_cap
            assert torch.equal(st.ovf[o:o + n], page.ovf[at[h]:at[h] + n]), h
            assert not bool(st.ovf[o + n:o + st.ovf_cap].any())                 # nothing behind a head's bytes
        assert not bool(st.ovf_used[:n_kv].any()) and not bool(st.ovf_used[2 * n_kv:].any()) and not bool(st.ovf[:n_kv * st.ovf_cap].any())
    assert room != 100 or cache.k.ovf_cap > small
    assert cache.S[heads].tolist() == [16 * tiles] * n_kv and cache.tail_len[heads].tolist() == [L % 16] * n_kv
