"""Bit-exact check of the BF16 rebuild that runs INSIDE the fused attention kernels.

The attention kernels decode compressed tiles straight into tensor-core fragments; nothing of the rebuilt K and V is normally
visible except through a softmax-weighted sum, where one wrong exponent among millions of elements would drown.  The library
therefore carries a second instantiation of the same kernels (gaac_debug_*_rebuild) that also writes every fragment word it
rebuilt to memory.  Here those words are compared bit for bit with what was encoded, over everything the kernels distinguish:
the three tiers, tiles whose escape bytes exceed the staged window (read from global memory instead), every byte phase of a
head's escape stream against the 16-byte copy granule, the raw BF16 tail of the slot layout with 1, 7 and 15 rows, and in the
paged layout small and large escape slots, finalized tiles that stayed raw, and the still-filling block.
"""
import numpy as np
import pytest
from common import to_bf16_cuda, bits, assert_attention_close
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu
SCALE = 128 ** -0.5
SENTINEL = 0x7FC1            # a NaN pattern no input contains: rows the kernel must not write keep it


def _junk_tiles(rng, n_heads, n_tok):
    """Random bit patterns (every group raw: 1280 escape bytes per tile), Inf/NaN and huge magnitudes removed."""
    junk = rng.integers(0, 65536, (n_heads, n_tok, 128)).astype(np.uint16)
    return np.where(((junk >> 7) & 0xFF) >= 0x86, junk & ~np.uint16(0x4000), junk)


def _rebuild_pages(kp, vp, q16, B, n_kv, G, nsplit):
    """Run the debug instantiation over two Pages -> (k_rebuilt, v_rebuilt) uint16 [B*n_kv, S_pad + 16, 128], fp32 output."""
    import torch
    from gaac_b200 import _lib
    from gaac_b200.kernel import _page_side, workspace
    n_q, S, S_pad = n_kv * G, kp.S, kp.sm.shape[1] // 128
    rows = S_pad + 16
    kr = torch.full((B * n_kv, rows, 128), SENTINEL, dtype=torch.int16, device="cuda"); vr = kr.clone()
    out = torch.empty(B, n_q, 128, dtype=torch.bfloat16, device="cuda"); o32 = torch.empty(B, n_q, 128, dtype=torch.float32, device="cuda")
    ws = workspace(torch.device("cuda"), B, n_q, nsplit)
    q = to_bf16_cuda(q16)
    rc = _lib.lib().gaac_debug_decode_attn_rebuild(_page_side(kp), _page_side(vp), q.data_ptr(), None, B, n_q, n_kv, None, S, S_pad,
                                                   SCALE, nsplit, None, 0, kp.base3.size(0), ws.data_ptr(), ws.numel(), out.data_ptr(), o32.data_ptr(),
                                                   kr.data_ptr(), vr.data_ptr(), rows, _lib.stream_ptr(torch.device("cuda")))
    assert rc == 0, rc
    torch.cuda.synchronize()
    return kr.cpu().numpy().view(np.uint16), vr.cpu().numpy().view(np.uint16), o32


def _assert_rebuilt(got, want16, S, what):
    """got [H, rows, 128] against the encoder's input want16 [H, S, 128]; rows >= S must be untouched."""
    bad = np.argwhere(got[:, :S] != want16)
    assert bad.size == 0, (what, "first mismatch (head, token, channel)", bad[0].tolist(), hex(int(got[tuple(bad[0])])), hex(int(want16[tuple(bad[0])])))
    assert (got[:, S:] == SENTINEL).all(), (what, "rows beyond the sequence were written")


@pytest.mark.parametrize("B,n_kv,G,S,nsplit", [(1, 2, 4, 1000, 3), (2, 2, 8, 333, 1), (1, 8, 4, 4096, 6), (3, 1, 1, 16, 1)])
def test_rebuild_inside_attention_is_bit_exact_all_tiers(B, n_kv, G, S, nsplit):
    import torch
    from gaac_b200 import Codec, TileEncoder
    rng = np.random.default_rng(S + G)
    k16, v16 = O.synth_kv("k", B * n_kv, S, 3, raw_frac=0.01, four_frac=0.2), O.synth_kv("v", B * n_kv, S, 4, raw_frac=0.01, four_frac=0.2)
    if S >= 333:                                           # two stretches of random bit patterns: their tiles overflow the staged window
        k16[:, 64:128] = _junk_tiles(rng, B * n_kv, 64); v16[:, 32:80] = _junk_tiles(rng, B * n_kv, 48)
    k, v = to_bf16_cuda(k16), to_bf16_cuda(v16)
    kp, vp = TileEncoder("k").encode(Codec(n_kv).calibrate(k), k), TileEncoder("v").encode(Codec(n_kv).calibrate(v), v)
    shares = O.tier_shares(kp.flags.cpu().numpy(), S)
    assert min(shares) > 0, shares                          # all three tiers occur
    q16 = O.f32_to_bf16((rng.standard_normal((B, n_kv * G, 128)) * 0.05).astype(np.float32))
    kr, vr, o32 = _rebuild_pages(kp, vp, q16, B, n_kv, G, nsplit)
    _assert_rebuilt(kr, k16, S, "K"); _assert_rebuilt(vr, v16, S, "V")
    for b in range(B):                                     # the debug instantiation computes the same attention
        assert_attention_close(o32[b].cpu().numpy(), q16[b], k16[b * n_kv:(b + 1) * n_kv].transpose(1, 0, 2), v16[b * n_kv:(b + 1) * n_kv].transpose(1, 0, 2), SCALE, b)


def test_rebuild_at_every_phase_of_the_escape_stream():
    """The escape window of a tile is copied from the 16-byte boundary below its first byte.  Shift the heads' escape bytes by
    0..15 bytes (head_start moves, the bytes stay the same) so that every alignment of a head's stream occurs."""
    import torch
    from gaac_b200 import Codec, TileEncoder
    n_kv, G, S = 2, 4, 512
    rng = np.random.default_rng(1)
    k16, v16 = O.synth_kv("k", n_kv, S, 13, raw_frac=0.02, four_frac=0.3), O.synth_kv("v", n_kv, S, 14, raw_frac=0.02, four_frac=0.3)
    k, v = to_bf16_cuda(k16), to_bf16_cuda(v16)
    kp, vp = TileEncoder("k").encode(Codec(n_kv).calibrate(k), k), TileEncoder("v").encode(Codec(n_kv).calibrate(v), v)
    q16 = O.f32_to_bf16((rng.standard_normal((1, n_kv * G, 128)) * 0.05).astype(np.float32))
    ovf_k, ovf_v, hs_k, hs_v = kp.ovf, vp.ovf, kp.ovf_head_start, vp.ovf_head_start
    for pad in range(16):
        for pg, ovf, hs in ((kp, ovf_k, hs_k), (vp, ovf_v, hs_v)):
            pg.ovf = torch.cat([torch.full((pad,), 0xEE, dtype=torch.uint8, device="cuda"), ovf]).contiguous()
            pg.ovf_head_start = (hs + pad).contiguous()
            if hasattr(pg, "_attn_side"): del pg._attn_side
        kr, vr, _ = _rebuild_pages(kp, vp, q16, 1, n_kv, G, 2)
        _assert_rebuilt(kr, k16, S, ("K", pad)); _assert_rebuilt(vr, v16, S, ("V", pad))


@pytest.mark.parametrize("tail", [1, 7, 15])
def test_rebuild_slot_cache_with_tail(tail):
    """Slot layout through the serving cache: compressed tiles of three sequences (one with per-sequence padding row -1) plus
    raw BF16 tails of `tail` rows, read through the slot map and the per-head length tables."""
    import torch
    from gaac_b200 import CompressedKVCache, _lib
    from gaac_b200.kernel import _side, workspace
    n_kv, G, n_slots = 2, 4, 3
    cache = CompressedKVCache(n_slots=n_slots, n_kv=n_kv, capacity=512)
    hist = {}
    for s, L in ((0, 64 + tail), (2, 160 + tail)):
        k16 = np.ascontiguousarray(O.synth_kv("k", n_kv, L, 20 + s, raw_frac=0.01).transpose(1, 0, 2))
        v16 = np.ascontiguousarray(O.synth_kv("v", n_kv, L, 30 + s, raw_frac=0.01).transpose(1, 0, 2))
        cache.prefill(s, to_bf16_cuda(k16), to_bf16_cuda(v16)); hist[s] = (k16, v16)
    slots_l = [2, -1, 0]
    B, n_q, rows = len(slots_l), n_kv * G, 512 + 16
    slots = torch.tensor(slots_l, dtype=torch.int32, device="cuda")
    q16 = O.f32_to_bf16((np.random.default_rng(tail).standard_normal((B, n_q, 128)) * 0.05).astype(np.float32))
    kr = torch.full((B * n_kv, rows, 128), SENTINEL, dtype=torch.int16, device="cuda"); vr = kr.clone()
    out = torch.empty(B, n_q, 128, dtype=torch.bfloat16, device="cuda")
    K, V = cache.k, cache.v
    sk = _side(K.sm, K.codes, K.flags, K.tile_off, K.ovf, K.head_start, K.base3, K.base4, K.tail)
    sv = _side(V.sm, V.codes, V.flags, V.tile_off, V.ovf, V.head_start, V.base3, V.base4, V.tail)
    ws = workspace(torch.device("cuda"), B, n_q, 2)
    q = to_bf16_cuda(q16)
    rc = _lib.lib().gaac_debug_decode_attn_rebuild(sk, sv, q.data_ptr(), slots.data_ptr(), B, n_q, n_kv, cache.S.data_ptr(), 0, cache.cap,
                                                   SCALE, 2, cache.tail_len.data_ptr(), 16, K.base3.shape[0], ws.data_ptr(), ws.numel(), out.data_ptr(), None,
                                                   kr.data_ptr(), vr.data_ptr(), rows, _lib.stream_ptr(torch.device("cuda")))
    assert rc == 0, rc
    torch.cuda.synchronize()
    kr, vr = kr.cpu().numpy().view(np.uint16), vr.cpu().numpy().view(np.uint16)
    for b, s in enumerate(slots_l):
        got_k, got_v = kr[b * n_kv:(b + 1) * n_kv], vr[b * n_kv:(b + 1) * n_kv]
        if s < 0:
            assert (got_k == SENTINEL).all() and (got_v == SENTINEL).all() and float(out[b].abs().max()) == 0.0
            continue
        k16, v16 = hist[s]
        _assert_rebuilt(got_k, k16.transpose(1, 0, 2), k16.shape[0], ("K", s)); _assert_rebuilt(got_v, v16.transpose(1, 0, 2), v16.shape[0], ("V", s))


@pytest.mark.parametrize("ovf_slot,adv,gen", [(128, 3, {}), (16, 0, dict(raw_frac=0.0, four_frac=0.004)), (128, 0, dict(raw_frac=0.02, four_frac=0.3))])
def test_rebuild_paged_layout(ovf_slot, adv, gen):
    """Paged layout: compressed slots with a 128-byte and a 16-byte escape area, finalized tiles that stayed raw (escapes did not
    fit, or adversarial bit patterns) and the filling block of every sequence, all read through block table and mode table."""
    import torch
    from gaac_b200 import _lib
    from gaac_b200.kernel import workspace
    from test_paged_gpu import _build_paged
    n_kv, G = 2, 4
    seq_lens = [16, 37, 333, 1000, 5]
    st, buf, bt, ks, vs = _build_paged(seq_lens, n_kv, 256, seed=21 + ovf_slot, adversarial_every=adv, ovf_slot=ovf_slot, raw_tiles=512, **gen)
    assert int(st.err) == 0                                           # the raw pool was large enough for every tile that stayed raw
    mt = st.mt.cpu().numpy()
    full_tiles = sum(L // 16 for L in seq_lens) * 2 * n_kv
    n_raw_final = int((mt < 0).sum()) - sum(1 for L in seq_lens if L % 16) * 2 * n_kv
    assert 0 < n_raw_final < full_tiles or (ovf_slot == 128 and adv == 0), (n_raw_final, full_tiles)     # both kinds of finalized tile occur
    B, n_q, rows = len(seq_lens), n_kv * G, 1024
    q16 = O.f32_to_bf16((np.random.default_rng(2).standard_normal((B, n_q, 128)) * 0.05).astype(np.float32))
    kr = torch.full((B * n_kv, rows, 128), SENTINEL, dtype=torch.int16, device="cuda"); vr = kr.clone()
    out = torch.empty(B, n_q * 128, dtype=torch.bfloat16, device="cuda")
    sl = torch.tensor(seq_lens, dtype=torch.int32, device="cuda")
    q = to_bf16_cuda(q16)
    for nsplit in (1, 3):
        kr.fill_(SENTINEL); vr.fill_(SENTINEL)
        ws = workspace(torch.device("cuda"), B, n_q, nsplit)
        rc = _lib.lib().gaac_debug_paged_decode_attn_rebuild(st.c_state(buf), bt.data_ptr(), bt.stride(0), sl.data_ptr(), q.data_ptr(), B, n_q,
                                                             SCALE, nsplit, ws.data_ptr(), ws.numel(), out.data_ptr(), None, kr.data_ptr(), vr.data_ptr(), rows,
                                                             _lib.stream_ptr(torch.device("cuda")))
        assert rc == 0, rc
        torch.cuda.synchronize()
        gk, gv = kr.cpu().numpy().view(np.uint16), vr.cpu().numpy().view(np.uint16)
        for b, L in enumerate(seq_lens):
            _assert_rebuilt(gk[b * n_kv:(b + 1) * n_kv], ks[b].transpose(1, 0, 2), L, ("K", b, nsplit))
            _assert_rebuilt(gv[b * n_kv:(b + 1) * n_kv], vs[b].transpose(1, 0, 2), L, ("V", b, nsplit))


def _tiles_with_raw_groups(kind, heads, counts, promoted, seed):
    """[heads, 16 * len(counts), 128]: tile i has counts[i] raw groups, a share `promoted` of the others is promoted; for base tables of 120 and 116 everywhere."""
    rng = np.random.default_rng(seed)
    e = rng.integers(120, 128, (heads, len(counts), 16 * 16, 8))                # in stored order: [tile][group of a row], 8 elements
    tier = np.where(rng.random(e.shape[:3]) < promoted, 1, 0)
    for h in range(heads):
        for i, n in enumerate(counts):
            tier[h, i, rng.permutation(256)[:n]] = 2
    at = rng.integers(0, 8, tier.shape)[..., None]
    low = np.where(tier == 2, 90, np.where(tier == 1, 117, 120))[..., None]
    np.put_along_axis(e, at, np.where(tier[..., None] > 0, low, np.take_along_axis(e, at, -1)), -1)
    x = (e << 7 | rng.integers(0, 128, e.shape) | rng.integers(0, 2, e.shape) << 15).astype(np.uint16).reshape(heads, -1, 128)
    out = np.empty_like(x)
    out[..., O.perm(kind)] = x                                                   # stored position i holds channel perm[i]
    return out


def _flat_bases(n_kv):
    import torch
    return torch.full((n_kv, 128), 120, dtype=torch.uint8), torch.full((n_kv, 128), 116, dtype=torch.uint8)


# raw groups of a tile pair around the 64 that have entries, on one side and on both; promoted groups among and behind them
@pytest.mark.parametrize("promoted", [0.0, 0.3])
def test_rebuild_with_as_many_raw_groups_as_have_room(promoted):
    import torch
    from gaac_b200 import Codec
    n_kv, G = 2, 4
    ck = [63, 64, 65, 0, 0, 0, 32, 32, 31, 1, 40, 20, 0, 256, 30, 3]
    cv = [0, 0, 0, 63, 64, 65, 31, 32, 34, 63, 23, 45, 0, 4, 256, 3]
    S = 16 * len(ck)
    k16, v16 = _tiles_with_raw_groups("k", n_kv, ck, promoted, 1), _tiles_with_raw_groups("v", n_kv, cv, promoted, 2)
    kp, vp = (Codec(n_kv).set_bases(*_flat_bases(n_kv)).encode(to_bf16_cuda(x), c) for x, c in ((k16, "k"), (v16, "v")))
    assert [int(n) for n in ((kp.flags.cpu().numpy().view(np.uint32)[..., None] >> np.arange(1, 32, 2, dtype=np.uint32)) & 1).reshape(n_kv, -1, 256).sum(-1)[0]] == ck
    q16 = O.f32_to_bf16((np.random.default_rng(3).standard_normal((1, n_kv * G, 128)) * 0.3).astype(np.float32))
    for nsplit in (1, 3):
        kr, vr, o32 = _rebuild_pages(kp, vp, q16, 1, n_kv, G, nsplit)
        _assert_rebuilt(kr, k16, S, ("k", nsplit))
        _assert_rebuilt(vr, v16, S, ("v", nsplit))
        assert_attention_close(o32[0].cpu().numpy(), q16[0], np.ascontiguousarray(k16.transpose(1, 0, 2)), np.ascontiguousarray(v16.transpose(1, 0, 2)), SCALE, nsplit)


@pytest.mark.parametrize("promoted", [0.0, 0.3])
def test_head_dim_256_with_as_many_raw_groups_as_have_room(promoted):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    from gaac_b200.vllm.paged_kernel256 import paged_attention256
    ck, cv = [55, 56, 57, 0, 0, 28, 28, 64, 5], [0, 0, 0, 56, 57, 28, 29, 4, 5]
    L, slot = 16 * len(ck), 528
    ks, vs = (np.ascontiguousarray(_tiles_with_raw_groups(c, 2, n, promoted, s).transpose(1, 0, 2)) for c, n, s in (("k", ck, 1), ("v", cv, 2)))
    b3, b4 = _flat_bases(2)
    st = LayerState(len(ck), 2, raw_tiles=8, bases=dict(k3=b3, k4=b4, v3=b3, v4=b4), ovf_slot=slot, device="cuda")
    buf = torch.zeros(len(ck) * 4 * (OVF_OFF + slot), dtype=torch.uint8, device="cuda")
    ent = torch.tensor([[t, 16 * t, 0, 16] for t in range(len(ck))], dtype=torch.int32, device="cuda")
    st.store(to_bf16_cuda(ks), to_bf16_cuda(vs), buf, ent, torch.empty(len(ck) * 4, dtype=torch.int32, device="cuda"))
    assert int(st.err) == 0 and (st.mt >= 0).all()
    for G in (4, 8):
        q16 = O.f32_to_bf16((np.random.default_rng(G).standard_normal((1, G, 256)) * 0.3).astype(np.float32))
        out, o32 = torch.empty(1, G * 256, dtype=torch.bfloat16, device="cuda"), torch.empty(1, G, 256, dtype=torch.float32, device="cuda")
        paged_attention256(to_bf16_cuda(q16), out, buf, st.raw, st.mt, torch.arange(len(ck), dtype=torch.int32, device="cuda")[None], torch.tensor([L], dtype=torch.int32, device="cuda"), st.bases,
                           st.TS, G, 1, out_f32=o32)
        assert_attention_close(o32[0].cpu().numpy(), q16[0], ks.reshape(L, 1, 256), vs.reshape(L, 1, 256), 256 ** -0.5, G)


def test_promoted_groups_take_no_room_from_raw_ones():
    """22 raw groups a side and a third of the others promoted: the entries suffice, and the kernel is as fast as with the raw groups alone (43 us of which 32768 tokens
    of 8 kv heads take 61 when their tiles go the way of those that have no room)."""
    import torch
    from gaac_b200 import Codec, attention
    n_kv, tiles = 8, 2048
    pages = {}
    for name, raw, promoted in (("room", 22, 0.33), ("none", 34, 0.33)):
        cols = [_tiles_with_raw_groups(c, 1, [raw] * 64, promoted, s) for c, s in (("k", 1), ("v", 2))]
        pages[name] = [Codec(n_kv).set_bases(*_flat_bases(n_kv)).encode(to_bf16_cuda(x).repeat(n_kv, tiles // 64, 1), c) for x, c in zip(cols, "kv")]
    q = torch.randn(1, 4 * n_kv, 128, device="cuda").to(torch.bfloat16)
    best = {}
    for name in list(pages) * 10:
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        attention(q, *pages[name])
        a.record()
        for _ in range(5): attention(q, *pages[name])
        b.record()
        torch.cuda.synchronize()
        best[name] = min(best.get(name, 1e9), a.elapsed_time(b) * 200)
    assert best["room"] < 0.85 * best["none"], best
