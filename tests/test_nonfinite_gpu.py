"""Attention over V with infinite and NaN elements: such an element makes its own channel infinite or NaN and leaves every other channel what it is without it.
Every place an element can be decoded from: the three tiers, tiles that the decoder reads from global memory, raw tiles, the filling block, the slot
tail, partial tiles, both halves of a 256-dim head."""
import numpy as np
import pytest
from common import to_bf16_cuda
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu
INF, NEG, NAN = 0x7F80, 0xFF80, 0x7FC1
CH = [5, 40, 100, 77]                                # channels that get such elements; 13, 32, 108 and 69, eight away from them, get none


def _plant(v16, rows, h=0, ch=CH):
    """v16 [L, heads, D]: Inf, -Inf and NaN at three rows, and a channel that has both infinities."""
    a, b, c, d = rows
    v16[a, h, ch[0]], v16[b, h, ch[1]], v16[c, h, ch[2]], v16[a, h, ch[3]], v16[d, h, ch[3]] = INF, NEG, NAN, INF, NEG


def _check(o32, q16, k16, v16, what):
    """o32 [n_q, D] against the oracle with the non-finite elements of V [L, n_kv, D] replaced by zeros, and their own channels."""
    n_q, n_kv = q16.shape[0], k16.shape[1]
    bad = (v16 & 0x7F80) == 0x7F80
    ref, mag = O.attention_ref(q16, k16, np.where(bad, np.uint16(0), v16), q16.shape[1] ** -0.5, with_abs=True)
    with np.errstate(invalid="ignore"):
        own = np.where(bad, O.bf16_to_f64(v16), 0.0).sum(0).repeat(n_q // n_kv, axis=0)                  # [n_q, D]: 0, +-Inf or NaN
    hit = bad.any(0).repeat(n_q // n_kv, axis=0)
    o = o32.astype(np.float64)
    assert np.array_equal(np.isnan(o), hit & np.isnan(own)), (what, "NaN at", np.argwhere(np.isnan(o) != (hit & np.isnan(own)))[:4])
    assert np.array_equal(o[hit & ~np.isnan(own)], own[hit & ~np.isnan(own)]), (what, "infinities")
    err = np.abs(np.where(hit, 0.0, o - ref)) / O.attention_bound(mag)
    assert err.max() <= 1.0, (what, err.max())


def _q(B, n_q, dim=128):
    return O.f32_to_bf16((np.random.default_rng(0).standard_normal((B, n_q, dim)) * 0.1).astype(np.float32))


def _k(heads, L, seed):
    """no outliers: a weight that underflows would make 0 x Inf, which is NaN in fp32 and Inf in the oracle's arithmetic"""
    return O.kv_like(heads, L, seed, outliers=0.0)


@pytest.mark.parametrize("mode", ["raw", "window3", "window4", "long"])
@pytest.mark.parametrize("n_kv,G,S", [(2, 4, 333), (1, 8, 1500), (1, 1, 16)])
def test_pages(mode, n_kv, G, S):
    import torch
    from gaac_b200 import Codec, attention
    k16, v16 = _k(n_kv, S, 3), O.kv_like(n_kv, S, seed=4)
    ck = Codec(n_kv).calibrate(to_bf16_cuda(k16))
    b3, b4 = O.calibrate(v16, n_kv)
    if mode == "long":                               # random bits, magnitudes moderate: more escape bytes than a stage holds
        junk = np.random.default_rng(S).integers(0, 65536, (n_kv, min(S, 96), 128)).astype(np.uint16)
        v16[:, :96] = np.where(((junk >> 7) & 0xFF) >= 0x86, junk & ~np.uint16(0x4000), junk)
    if mode.startswith("window"):                    # channels whose window ends at exponent 255
        v16[:, :, CH] = (v16[:, :, CH] & 0x807F) | np.uint16(249 << 7)
        b3[:, CH] = 248 if mode == "window3" else 100
        b4[:, CH] = 240
    vt = np.ascontiguousarray(v16.transpose(1, 0, 2))
    _plant(vt, [3, 14, S - 1, 7] if S == 16 else [3, 19, S - 1, 50])
    kp, vp = ck.encode(to_bf16_cuda(k16), "k"), Codec(n_kv).set_bases(torch.from_numpy(b3), torch.from_numpy(b4)).encode(to_bf16_cuda(np.ascontiguousarray(vt.transpose(1, 0, 2))), "v")
    q16 = _q(1, n_kv * G)
    for nsplit in (None, 1, 3):
        o32 = torch.empty(1, n_kv * G, 128, dtype=torch.float32, device="cuda")
        attention(to_bf16_cuda(q16), kp, vp, nsplit=nsplit, out_f32=o32)
        _check(o32[0].cpu().numpy(), q16[0], np.ascontiguousarray(k16.transpose(1, 0, 2)), vt, (mode, nsplit))


@pytest.mark.parametrize("n_kv,G", [(2, 4), (1, 6)])
@pytest.mark.parametrize("nsplit", [None, 1, 4])
def test_slots_with_tails(n_kv, G, nsplit):
    import torch
    from gaac_b200 import CompressedKVCache
    lens = [700, 13, 300, 77]
    cache = CompressedKVCache(n_slots=4, n_kv=n_kv, capacity=1024, bases=None)
    hist = []
    for s, L in enumerate(lens):
        k, v = (np.ascontiguousarray(f(n_kv, L, 7 * s + i).transpose(1, 0, 2)) for i, f in ((1, _k), (2, O.kv_like)))
        if s != 2:                                   # row 2 stays finite: nothing of its neighbours reaches it
            _plant(v, [L - 1, L - 2, 2, 5] if s else [500, 33, L - 1, 80], h=n_kv - 1)
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v), check=False)
        hist.append((k, v))
    q16 = _q(4, n_kv * G)
    o32 = torch.empty(4, n_kv * G, 128, dtype=torch.float32, device="cuda")
    cache.attention(to_bf16_cuda(q16), torch.arange(4, dtype=torch.int32, device="cuda"), 128 ** -0.5, nsplit=nsplit, max_len=700, out_f32=o32)
    for b in range(4):
        _check(o32[b].cpu().numpy(), q16[b], *hist[b], (b, nsplit))


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n_kv,G", [(2, 4), (1, 7)])
@pytest.mark.parametrize("nsplit", [None, 1, 4])
def test_paged(wide, n_kv, G, nsplit):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    from gaac_b200.vllm.paged_kernel import paged_attention
    from gaac_b200.vllm.paged_kernel256 import paged_attention256
    heads, dim = (2 * n_kv, 256) if wide else (n_kv, 128)
    stored, lens = [16, 605, 1210, 40], [16, 605, 1201, 30]                  # the last two: rows behind the end, in compressed tiles and in the filling block
    ends = np.cumsum(stored)
    ks, vs = ([np.ascontiguousarray(x[:, e - L:e].transpose(1, 0, 2)) for e, L in zip(ends, stored)] for x in (_k(heads, ends[-1], 1), O.kv_like(heads, ends[-1], 2)))
    junk = np.random.default_rng(1).integers(0, 65536, (16, heads, 128)).astype(np.uint16)
    vs[1][32:48] = np.where(((junk >> 7) & 0xFF) >= 0x86, junk & ~np.uint16(0x4000), junk)                # a block of V that stays raw
    _plant(vs[1], [34, 47, 604, 601], h=heads - 1)   # raw tile, filling block
    _plant(vs[2], [100, 1000, 1199, 17], h=0)
    vs[2][1203:, :, 9] = INF                         # behind the end: not part of the sequence
    vs[3][31:, :, 9] = NAN
    bases = {}
    for kind, xs in (("k", ks), ("v", vs)):
        bases[kind + "3"], bases[kind + "4"] = (torch.from_numpy(b) for b in O.calibrate(np.ascontiguousarray(xs[2].transpose(1, 0, 2)), heads))
    need = [-(-L // 16) for L in stored]
    st = LayerState(sum(need), heads, raw_tiles=2 * sum(need) * heads, bases=bases, ovf_slot=128, device="cuda")
    buf = torch.zeros(sum(need) * 2 * heads * (OVF_OFF + 128), dtype=torch.uint8, device="cuda")
    bt, first = np.zeros((4, max(need)), np.int32), 0
    for i, L in enumerate(stored):
        bt[i, :need[i]] = np.arange(first, first + need[i]); first += need[i]
        ent = torch.tensor([[bt[i, t], 16 * t, 0, min(16, L - 16 * t)] for t in range(need[i])], dtype=torch.int32, device="cuda")
        st.store(to_bf16_cuda(ks[i]), to_bf16_cuda(vs[i]), buf, ent, torch.empty(need[i] * 2 * heads, dtype=torch.int32, device="cuda"))
    assert int(st.err) == 0 and (st.mt.view(-1, heads, 2)[bt[1, 2], :, 1] < 0).all()
    n_q = n_kv * G
    q16 = _q(4, n_q, dim)
    out = torch.empty(4, n_q * dim, dtype=torch.bfloat16, device="cuda")
    o32 = torch.empty(4, n_q, dim, dtype=torch.float32, device="cuda")
    (paged_attention256 if wide else paged_attention)(to_bf16_cuda(q16), out, buf, st.raw, st.mt, torch.from_numpy(bt).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), st.bases,
                                                      st.TS, n_q, n_kv, nsplit, out_f32=o32)
    for b in range(4):
        _check(o32[b].cpu().numpy(), q16[b], ks[b][:lens[b]].reshape(lens[b], n_kv, dim), vs[b][:lens[b]].reshape(lens[b], n_kv, dim), (b, nsplit))
