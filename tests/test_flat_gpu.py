"""One wave of CTAs over the tiles of all rows and kv heads (gaac_decode_attn_flat, gaac_paged_decode_attn_flat): every row against the fp64 oracle, with one CTA
for everything, a few, as many as there are SMs and more than there are tiles; empty rows, rows that are all tail, padding rows, 1 to 2049 rows; V
elements that are not finite (their CTA repeats its piece)."""
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O
from test_paged_gpu import _build_paged

SCALE = 128 ** -0.5


def test_choose_flat_bounds():
    from gaac_b200.kernel import choose_flat, choose_nsplit_sm100, choose_units
    for n_kv in (1, 2, 8, 148, 149):
        for B in (1, 2, 7, 33, 64, 300, 1025):
            for S in (1, 300, 5000, 10 ** 6):
                units = choose_units(B, n_kv, S)
                flat = choose_flat(B, n_kv, S, choose_nsplit_sm100(B, n_kv, S), units)
                assert flat in (0, 148) and not (flat and (B == 1 or S <= 2544))
    assert choose_flat(64, 1, 32769, 9, 0) == 148 and choose_flat(148, 1, 1000, 1, 0) == 0


@pytest.mark.parametrize("B,cap", [(64, 32768), (1024, 1 << 20), (1024, 1 << 25), (4096, 1 << 22), (4096, 1 << 23)])
def test_flat_launches_are_chosen_where_the_library_takes_them(monkeypatch, B, cap):
    """max_len only steers the choice: a cache whose capacity is so large that the line of a flat launch could not be counted gets another form, not a refusal."""
    import ctypes, types
    import torch
    import gaac_b200.kv_cache as kvc
    from gaac_b200 import _lib
    cache = object.__new__(kvc.CompressedKVCache)
    store = types.SimpleNamespace(**{n: None for n in ("sm", "codes", "flags", "tile_off", "ovf", "head_start", "base3", "base4", "tail")})
    cache.n_kv, cache.cap, cache.k, cache.v, cache._pending, cache.S, cache.tail_len = 1, cap, store, store, {}, None, None
    seen = []
    monkeypatch.setattr(kvc, "_ext", lambda: types.SimpleNamespace(gaac_attn_launch=lambda *a, flat, **k: (seen.append(flat), a[16])[1]))
    fake, side = ctypes.c_void_p(0x1000), _lib.Side(0x1000, 0x1000, 0x1000, 0x1000, 0x1000, 0x1000, 64, 0x1000, 0x1000, None)
    for max_len in (3000, 8192, None):
        cache.attention(torch.zeros(B, 4, 128, dtype=torch.bfloat16), torch.zeros(B, dtype=torch.int32), SCALE, max_len=max_len)
        if seen[-1]:                                                            # 5: only the workspace is too small
            assert _lib.lib().gaac_decode_attn_flat(side, side, fake, fake, B, 4, 1, fake, cap, 0.1, seen[-1], None, 0, 1, fake, 64, fake, None, None) == 5
    assert any(seen) == (B * (cap // 16 + 64) < 1 << 30)


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G,lens", [(2, 4, [0, 5, 16, 1000, 17]), (1, 8, [700]), (2, 1, [333] * 6), (3, 5, [3, 33, 64, 65, 900, 1, 0, 300, 15, 16, 31, 47, 48, 49] * 5)])
def test_slots_flat(monkeypatch, n_kv, G, lens):
    import torch
    import gaac_b200.kv_cache as kvc
    B, hist = len(lens), {}
    cache = kvc.CompressedKVCache(n_slots=B, n_kv=n_kv, capacity=1024, bases=None)
    for s, L in enumerate(lens):
        k, v = (np.ascontiguousarray(O.kv_like(n_kv, max(L, 1), 7 * s + i).transpose(1, 0, 2))[:L] for i in (1, 2))
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v), check=False)
        hist[s] = (k, v)
    rng = np.random.default_rng(B)
    order = rng.permutation(B)
    order[B // 2] = -1 if B > 1 else order[B // 2]
    slots = torch.tensor(order, dtype=torch.int32, device="cuda")
    q16 = O.f32_to_bf16((rng.standard_normal((B, n_kv * G, 128)) * 0.1).astype(np.float32))
    for ctas in (1, 3, 37, 148, 148, 1000):                                     # the same call twice: the split counters are left at zero
        monkeypatch.setattr(kvc, "choose_flat", lambda *a, n=ctas: n)
        o32 = torch.empty(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
        out = cache.attention(to_bf16_cuda(q16), slots, SCALE, max_len=1000, out_f32=o32)
        for b, s in enumerate(order):
            if s < 0 or lens[s] == 0:
                assert not out[b].any(), (b, s, ctas)
            else:
                assert_attention_close(o32[b].cpu().numpy(), q16[b], *hist[s], SCALE, (b, s, ctas))


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G,lens", [(2, 4, [16, 37, 333, 1000, 5]), (1, 8, [1500, 1]), (4, 1, [1, 500] * 20)])
def test_paged_flat(monkeypatch, n_kv, G, lens):
    import torch
    import gaac_b200.vllm.paged_kernel as pk
    blocks = sum(-(-x // 16) for x in lens)
    st, buf, bt, ks, vs = _build_paged(lens, n_kv, blocks + 4, seed=n_kv, adversarial_every=5, raw_tiles=2 * n_kv * blocks)
    assert int(st.err) == 0
    B, n_q = len(lens), n_kv * G
    q16 = O.f32_to_bf16((np.random.default_rng(1).standard_normal((B, n_q, 128)) * 0.3).astype(np.float32))
    lens_now = list(lens)
    lens_now[B // 2] = 0                                                        # a row without tokens between others
    sl = torch.tensor(lens_now, dtype=torch.int32, device="cuda")
    for ctas in (1, 3, 37, 148, 1000):
        monkeypatch.setattr(pk, "choose_flat", lambda *a, n=ctas: n)
        o32 = torch.empty(B, n_q, 128, dtype=torch.float32, device="cuda")
        out = torch.full((B, n_q * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        pk.paged_attention(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_q, n_kv, out_f32=o32)
        for b in range(B):
            if lens_now[b] == 0:
                assert not out[b].any(), (b, ctas)
            else:
                assert_attention_close(o32[b].cpu().numpy(), q16[b], ks[b], vs[b], SCALE, (b, ctas))


@pytest.mark.gpu
def test_flat_pieces_with_infinite_elements(monkeypatch):
    import torch
    import gaac_b200.kv_cache as kvc
    n_kv, G, lens = 1, 4, [400, 90, 1000]
    cache = kvc.CompressedKVCache(n_slots=3, n_kv=n_kv, capacity=1024, bases=None)
    q16 = O.f32_to_bf16((np.random.default_rng(3).standard_normal((3, n_kv * G, 128)) * 0.1).astype(np.float32))
    for s, L in enumerate(lens):
        k, v = (np.ascontiguousarray(O.kv_like(n_kv, L, 9 * s + i, outliers=0.0).transpose(1, 0, 2)) for i in (1, 2))        # (no weight underflows: 0 x Inf is NaN)
        v[L // 2, 0, 5] = 0x7F80                                                # one infinite element of channel 5
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v))
    slots = torch.arange(3, dtype=torch.int32, device="cuda")
    want = cache.attention(to_bf16_cuda(q16), slots, SCALE, nsplit=2).float()
    for ctas in (1, 4, 148):
        monkeypatch.setattr(kvc, "choose_flat", lambda *a, n=ctas: n)
        got = cache.attention(to_bf16_cuda(q16), slots, SCALE, max_len=1000).float()
        assert torch.isinf(got[:, :, 5]).all() and torch.isfinite(got[:, :, :5]).all() and torch.isfinite(got[:, :, 6:]).all()
        keep = [c for c in range(128) if c != 5]
        assert torch.allclose(got[:, :, keep], want[:, :, keep], rtol=2 ** -7, atol=1e-3)        # BF16 results of the same sums in another order


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G", [(3, 4), (2, 6)])
@pytest.mark.parametrize("where", [None, 5, -3])
def test_heads_of_different_lengths(monkeypatch, n_kv, G, where):
    """A slot's first head is 64 and 320 tokens shorter, or 208 longer, than the others (a refused append leaves one head's counters alone); where: a row of the LAST head
    that holds an infinite element, which its CTA's repeat of the piece has to find as well."""
    import torch
    import gaac_b200.kv_cache as kvc
    cache = kvc.CompressedKVCache(n_slots=3, n_kv=n_kv, capacity=1024, bases=None)
    full, first, rest, hist = [640, 960, 800], [576, 640, 800], [640, 960, 592], []
    for s, L in enumerate(full):
        k, v = (np.ascontiguousarray(O.kv_like(n_kv, L, 9 * s + i, outliers=0.0).transpose(1, 0, 2)) for i in (1, 2))
        if where is not None: v[where % rest[s], n_kv - 1, 5] = 0x7F80
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v))
        cache.S[s * n_kv:(s + 1) * n_kv] = torch.tensor([first[s]] + [rest[s]] * (n_kv - 1))
        hist.append((k, v))
    q16 = O.f32_to_bf16((np.random.default_rng(n_kv).standard_normal((3, n_kv * G, 128)) * 0.1).astype(np.float32))
    slots = torch.arange(3, dtype=torch.int32, device="cuda")
    for ctas in (0, 1, 4, 37, 148):                                             # 0: the grid
        monkeypatch.setattr(kvc, "choose_flat", lambda *a, n=ctas: n)
        o32 = torch.empty(3, n_kv * G, 128, dtype=torch.float32, device="cuda")
        cache.attention(to_bf16_cuda(q16), slots, SCALE, max_len=1000, nsplit=None if ctas else 2, out_f32=o32)
        for b, (k, v) in enumerate(hist):
            for h in range(n_kv):
                L = rest[b] if h else first[b]
                got, vh = o32[b, h * G:(h + 1) * G].cpu().numpy(), v[:L, h:h + 1].copy()
                if where is not None and h == n_kv - 1:
                    assert np.isposinf(got[:, 5]).all(), (b, h, ctas)
                    vh[where % rest[b], 0, 5] = 0; got[:, 5] = 0
                    ref = O.attention_ref(q16[b, h * G:(h + 1) * G], k[:L, h:h + 1], vh, SCALE)
                    got[:, 5] = ref[:, 5]
                assert_attention_close(got, q16[b, h * G:(h + 1) * G], k[:L, h:h + 1], vh, SCALE, (b, h, ctas))


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("G", [4, 7])
def test_paged_pieces_with_infinite_elements(monkeypatch, wide, G):
    """The repeat of a piece in the paged forms: every channel without an infinite element against the fp64 oracle."""
    import torch
    import gaac_b200.vllm.paged_kernel as pk, gaac_b200.vllm.paged_kernel256 as pk256
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    dim, heads, lens = (256, 2, [700, 33, 1200]) if wide else (128, 1, [700, 33, 1200])
    need = [-(-L // 16) for L in lens]
    ks, vs = ([np.ascontiguousarray(O.kv_like(heads, L, 5 * i + s, outliers=0.0).transpose(1, 0, 2)) for i, L in enumerate(lens)] for s in (1, 2))
    bases = {}
    for kind, xs in (("k", ks), ("v", vs)):
        bases[kind + "3"], bases[kind + "4"] = (torch.from_numpy(b) for b in O.calibrate(np.ascontiguousarray(xs[2].transpose(1, 0, 2)), heads))
    for i, L in enumerate(lens):
        vs[i][L - 1, 0, 5] = vs[i][L // 2, heads - 1, 9] = 0x7F80
    st = LayerState(sum(need), heads, raw_tiles=2 * sum(need) * heads, bases=bases, ovf_slot=128, device="cuda")
    buf = torch.zeros(sum(need) * 2 * heads * (OVF_OFF + 128), dtype=torch.uint8, device="cuda")
    bt, at = np.zeros((3, max(need)), np.int32), 0
    for i, L in enumerate(lens):
        bt[i, :need[i]] = np.arange(at, at + need[i]); at += need[i]
        ent = torch.tensor([[bt[i, t], 16 * t, 0, min(16, L - 16 * t)] for t in range(need[i])], dtype=torch.int32, device="cuda")
        st.store(to_bf16_cuda(ks[i]), to_bf16_cuda(vs[i]), buf, ent, torch.empty(need[i] * 2 * heads, dtype=torch.int32, device="cuda"))
    assert int(st.err) == 0
    q16 = O.f32_to_bf16((np.random.default_rng(3).standard_normal((3, G, dim)) * 0.1).astype(np.float32))
    call = pk256.paged_attention256 if wide else pk.paged_attention
    for ctas in (1, 4, 148):
        monkeypatch.setattr(*((pk256, "choose_flat256") if wide else (pk, "choose_flat")), lambda *a, n=ctas: n)
        o32 = torch.empty(3, G, dim, dtype=torch.float32, device="cuda")
        out = torch.empty(3, G * dim, dtype=torch.bfloat16, device="cuda")
        call(to_bf16_cuda(q16), out, buf, st.raw, st.mt, torch.from_numpy(bt).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), st.bases, st.TS, G, 1, out_f32=o32)
        for b, L in enumerate(lens):
            k, v, got = ks[b].reshape(L, 1, dim), vs[b].reshape(L, 1, dim), o32[b].cpu().numpy()
            hit = ((v & 0x7FFF) == 0x7F80).any((0, 1))
            assert np.isposinf(got[:, hit]).all() and hit.sum() == 2, (b, ctas)
            v = np.where((v & 0x7FFF) == 0x7F80, np.uint16(0), v)
            got[:, hit] = O.attention_ref(q16[b], k, v, dim ** -0.5)[:, hit]
            assert_attention_close(got, q16[b], k, v, dim ** -0.5, (b, ctas))


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G,lens", [(2, 4, [16, 37, 333, 1000, 5]), (1, 8, [1500, 1]), (3, 1, [1, 260] * 17), (1, 6, [900])])
def test_paged256_flat(monkeypatch, n_kv, G, lens):
    import torch
    import gaac_b200.vllm.paged_kernel256 as pk
    blocks = sum(-(-x // 16) for x in lens)
    st, buf, bt, ks, vs = _build_paged(lens, 2 * n_kv, blocks + 4, seed=n_kv, adversarial_every=5, raw_tiles=4 * n_kv * blocks)
    assert int(st.err) == 0
    B, n_q = len(lens), n_kv * G
    q16 = O.f32_to_bf16((np.random.default_rng(1).standard_normal((B, n_q, 256)) * 0.3).astype(np.float32))
    lens_now = list(lens)
    if B > 1: lens_now[B // 2] = 0                                              # a row without tokens between others
    sl = torch.tensor(lens_now, dtype=torch.int32, device="cuda")
    for ctas in (1, 3, 37, 148, 148, 1000):
        monkeypatch.setattr(pk, "choose_flat256", lambda *a, n=ctas: n)
        o32 = torch.empty(B, n_q, 256, dtype=torch.float32, device="cuda")
        out = torch.full((B, n_q * 256), float("nan"), dtype=torch.bfloat16, device="cuda")
        pk.paged_attention256(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_q, n_kv, out_f32=o32)
        for b in range(B):
            L = lens_now[b]
            if L == 0:
                assert not out[b].any(), (b, ctas)
            else:
                assert_attention_close(o32[b].cpu().numpy(), q16[b], ks[b].reshape(-1, n_kv, 256)[:L], vs[b].reshape(-1, n_kv, 256)[:L], 256 ** -0.5, (b, ctas))


# Many rows over a few stored sequences.  Rows that are dealt out whole (1 to 32 pairs a CTA), too many rows for that (513), too many to be held while the plan is made
# (2049), more pairs than are dealt out (7 CTAs); one piece per CTA (1000 CTAs), rows of one length and of very different ones
@pytest.mark.gpu
@pytest.mark.parametrize("rows,short", [(40, True), (160, True), (160, False), (512, True), (513, True), (2049, False)])
@pytest.mark.parametrize("paged", [False, True])
def test_plans_of_many_rows(monkeypatch, rows, short, paged):
    import torch
    import gaac_b200.kv_cache as kvc, gaac_b200.vllm.paged_kernel as pk
    n_kv, G = 2, 4
    rng = np.random.default_rng(rows)
    lens = [int(x) for x in rng.integers(1, 260, 12)] + [16, 1, 0, 0] if short else [1500, 3, 40, 700, 16, 90, 0, 33]
    pick = rng.integers(0, len(lens), rows)
    pick[: len(lens)] = np.arange(len(lens))[: rows]
    q16 = O.f32_to_bf16((rng.standard_normal((len(lens), n_kv * G, 128)) * 0.1).astype(np.float32))
    q, idx = to_bf16_cuda(q16)[torch.from_numpy(pick)].contiguous(), torch.from_numpy(pick).cuda()
    if paged:
        full = [max(L, 1) for L in lens]
        st, buf, bt, ks, vs = _build_paged(full, n_kv, sum(-(-L // 16) for L in full) + 4, seed=3, raw_tiles=4 * n_kv * len(lens))
        sl = torch.tensor(lens, dtype=torch.int32, device="cuda")[idx]
        out, bt = torch.empty(rows, n_kv * G * 128, dtype=torch.bfloat16, device="cuda"), bt[idx].contiguous()
        call = lambda o32: pk.paged_attention(q, out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_kv * G, n_kv, out_f32=o32)
    else:
        ks, vs = ([np.ascontiguousarray(O.kv_like(n_kv, max(L, 1), 7 * i + s).transpose(1, 0, 2)) for i, L in enumerate(lens)] for s in (1, 2))
        cache = kvc.CompressedKVCache(n_slots=len(lens), n_kv=n_kv, capacity=1536, bases=None)
        for i, L in enumerate(lens):
            if L: cache.prefill(i, to_bf16_cuda(ks[i]), to_bf16_cuda(vs[i]), check=False)
        call = lambda o32: cache.attention(q, idx.int(), SCALE, max_len=1500, out_f32=o32)
    refs = [O.attention_ref(q16[i], ks[i][:L], vs[i][:L], SCALE, with_abs=True) for i, L in enumerate(lens)]
    ref = torch.from_numpy(np.stack([r for r, _ in refs])).cuda()
    bound = torch.from_numpy(np.stack([O.attention_bound(m) for _, m in refs])).cuda()
    for ctas in (7, 37, 148, 148, 1000):
        monkeypatch.setattr(kvc, "choose_flat", lambda *a, n=ctas: n)
        monkeypatch.setattr(pk, "choose_flat", lambda *a, n=ctas: n)
        o32 = torch.full((rows, n_kv * G, 128), float("nan"), dtype=torch.float32, device="cuda")
        call(o32)
        worst = ((o32.double() - ref[idx]).abs() / bound[idx]).amax((1, 2))
        assert bool((worst <= 1.0).all()), (ctas, [int(b) for b in (~(worst <= 1.0)).nonzero().ravel()[:8]])


@pytest.mark.gpu
def test_short_rows_in_a_wide_table_are_no_slower_than_in_a_narrow_one():
    """The launch that the rule picks for a table of 8192 tokens, rows of 100 to 400 tokens: the grid of a table that fits takes 32 us, pieces of equal shares of a line 40."""
    import torch
    import gaac_b200.vllm.paged_kernel as pk
    from gaac_b200.kernel import choose_flat
    B, n_kv, G = 64, 8, 4
    lens = [int(x) for x in np.random.default_rng(5).integers(100, 400, B)]
    st, buf, bt, ks, vs = _build_paged(lens, n_kv, sum(-(-L // 16) for L in lens) + 4, seed=3, raw_tiles=2 * n_kv * B + 64)
    wide = torch.nn.functional.pad(bt, (0, 512 - bt.shape[1])).contiguous()
    assert choose_flat(B, n_kv, 8192, 1, 0, G) == 148                           # reached through the rule itself
    q16 = O.f32_to_bf16((np.random.default_rng(1).standard_normal((B, n_kv * G, 128)) * 0.3).astype(np.float32))
    q, sl = to_bf16_cuda(q16), torch.tensor(lens, dtype=torch.int32, device="cuda")
    out, best = torch.empty(B, n_kv * G * 128, dtype=torch.bfloat16, device="cuda"), {}
    o32 = torch.empty(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
    call = lambda t, **k: pk.paged_attention(q, out, buf, st.raw, st.mt, t, sl, st.bases, st.TS, n_kv * G, n_kv, **k)
    call(wide, out_f32=o32)
    for b in (0, 17, B - 1):
        assert_attention_close(o32[b].cpu().numpy(), q16[b], ks[b], vs[b], SCALE, b)
    for name, table in (("narrow", bt), ("wide", wide)) * 10:
        a, e = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        call(table)
        a.record()
        for _ in range(20): call(table)
        e.record()
        torch.cuda.synchronize()
        best[name] = min(best.get(name, 1e9), a.elapsed_time(e) * 50)
    assert best["wide"] < 1.12 * best["narrow"], best


@pytest.mark.parametrize("flat,units,name", [(148, 0, "gaac_decode_attn_flat"), (0, 12, "gaac_decode_attn_balanced")])
def test_a_refused_call_is_reported_by_its_own_name(monkeypatch, flat, units, name):
    import types
    import torch
    from gaac_b200 import _lib, kernel
    monkeypatch.setattr(kernel, "workspace", lambda *a: torch.zeros(64, dtype=torch.uint8))
    monkeypatch.setattr(_lib, "stream_ptr", lambda dev=None: None)
    t, i = torch.zeros(16, 128, dtype=torch.uint8), torch.zeros(16, dtype=torch.int32)
    q = types.SimpleNamespace(size=lambda d: 128, is_cuda=True, device="cpu", dtype=torch.bfloat16, data_ptr=lambda: 16)
    with pytest.raises(RuntimeError, match=name + ":"):
        kernel._Ext.gaac_attn_launch(t, t, i, i, t, i, t, t, t, t, i, i, t, i, t, t, q, i[:4], 4, 1, i, 17, 0.1, None, t[:0], t[:0], i, 0, units=units, flat=flat)          # (a capacity of 17 tokens)
