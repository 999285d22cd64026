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
