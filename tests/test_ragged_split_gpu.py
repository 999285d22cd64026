"""Ragged batches whose rows share the GPU by their lengths (gaac_decode_attn_balanced, gaac_paged_decode_attn_balanced): every row against the fp64
oracle, for the fewest ranges, the most, and numbers in between; empty rows, rows that are all tail, padding rows, 1 to 32 rows."""
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O
from test_paged_gpu import _build_paged

SCALE = 128 ** -0.5


def test_choose_units_bounds():
    from gaac_b200.kernel import choose_units
    for n_kv in (1, 2, 4, 8, 32, 148, 149):
        for B in range(1, 66):
            for S in (0, 1, 64, 65, 5000, 10 ** 6):
                u = choose_units(B, n_kv, S)
                assert u == 0 or (B <= u and u * n_kv <= 148 and B <= 32 and u - B + 1 <= 1024)
    assert choose_units(1, 8, 4096) == 0 and choose_units(9, 8, 4096) == 18 and choose_units(9, 8, 20000) == 0 and choose_units(4, 8, 20000) == 18 and choose_units(10, 8, 4096) == 0 and choose_units(33, 1, 4096) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G,lens", [(2, 4, [0, 5, 16, 1000, 17]), (1, 8, [700]), (1, 5, [3, 33, 64, 65, 2000, 1, 0, 300, 15, 16, 31, 47, 48, 49, 63] * 2 + [900, 2])])
def test_slots_share_by_length(monkeypatch, n_kv, G, lens):
    import torch
    import gaac_b200.kv_cache as kvc
    B, hist = len(lens), {}
    cache = kvc.CompressedKVCache(n_slots=B, n_kv=n_kv, capacity=2048, bases=None)
    for s, L in enumerate(lens):
        k, v = (np.ascontiguousarray(O.kv_like(n_kv, max(L, 1), 7 * s + i).transpose(1, 0, 2))[:L] for i in (1, 2))
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v), check=False)
        hist[s] = (k, v)
    rng = np.random.default_rng(B)
    order = rng.permutation(B)
    order[B // 2] = -1 if B > 1 else order[B // 2]
    slots = torch.tensor(order, dtype=torch.int32, device="cuda")
    q16 = O.f32_to_bf16((rng.standard_normal((B, n_kv * G, 128)) * 0.1).astype(np.float32))
    for units in (B, B + 1, 2 * B + 3, 148 // n_kv, 148 // n_kv):              # the same call twice: the split counters are left at zero
        monkeypatch.setattr(kvc, "choose_units", lambda *a, u=units: u)
        o32 = torch.empty(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
        out = cache.attention(to_bf16_cuda(q16), slots, SCALE, max_len=2000, out_f32=o32)
        for b, s in enumerate(order):
            if s < 0 or lens[s] == 0:
                assert not out[b].any(), (b, s, units)
            else:
                assert_attention_close(o32[b].cpu().numpy(), q16[b], *hist[s], SCALE, (b, s, units))


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G,lens", [(2, 4, [16, 37, 333, 1000, 5]), (1, 8, [1500, 1]), (4, 1, [1, 500] * 16)])
def test_paged_rows_share_by_length(monkeypatch, n_kv, G, lens):
    import torch
    import gaac_b200.vllm.paged_kernel as pk
    blocks = sum(-(-x // 16) for x in lens)
    st, buf, bt, ks, vs = _build_paged(lens, n_kv, blocks + 4, seed=n_kv, adversarial_every=5, raw_tiles=2 * n_kv * blocks)
    assert int(st.err) == 0
    B, n_q = len(lens), n_kv * G
    q16 = O.f32_to_bf16((np.random.default_rng(1).standard_normal((B, n_q, 128)) * 0.3).astype(np.float32))
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    for units in (B, B + 1, 2 * B + 3, 148 // n_kv):
        monkeypatch.setattr(pk, "choose_units", lambda *a, u=units: max(u, B))
        out = torch.empty(B, n_q * 128, dtype=torch.bfloat16, device="cuda")
        o32 = torch.empty(B, n_q, 128, dtype=torch.float32, device="cuda")
        pk.paged_attention(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_q, n_kv, out_f32=o32)
        for b in range(B):
            assert_attention_close(o32[b].cpu().numpy(), q16[b], ks[b], vs[b], SCALE, (b, units))


def test_two_waves_only_where_one_is_mostly_idle():
    from gaac_b200.kernel import choose_units
    two = {(B, n, S) for n in (1, 2, 4, 8) for B in range(2, 33) for S in (1000, 4000, 8000, 12000, 16000, 30000) if choose_units(B, n, S) * n > 148}
    assert two == {(B, n, S) for n, rows in ((8, (7,)), (4, (13, 14)), (2, range(25, 30))) for B in rows for S in (12000, 16000)}
    assert all(choose_units(B, n, S) * n <= 296 for B, n, S in two)


# units of two waves: rows of equal length that fit a second wave better, and ragged ones whose CTAs behind the first wave find nothing to do
@pytest.mark.gpu
@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("lens", [[4100] * 7, [3000, 60, 4100, 0, 700, 16, 1999]])
def test_units_of_two_waves(monkeypatch, paged, lens):
    import torch
    import gaac_b200.kv_cache as kvc
    import gaac_b200.vllm.paged_kernel as pk
    n_kv, G, B = 8, 4, 7
    q16 = O.f32_to_bf16((np.random.default_rng(3).standard_normal((B, n_kv * G, 128)) * 0.1).astype(np.float32))
    o32 = torch.empty(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
    if paged:
        st, buf, bt, ks, vs = _build_paged([max(x, 1) for x in lens], n_kv, sum(-(-max(x, 1) // 16) for x in lens) + 4, seed=3)
        call = lambda: pk.paged_attention(to_bf16_cuda(q16), torch.empty(B, n_kv * G * 128, dtype=torch.bfloat16, device="cuda"), buf, st.raw, st.mt, bt,
                                          torch.tensor(lens, dtype=torch.int32, device="cuda"), st.bases, st.TS, n_kv * G, n_kv, out_f32=o32)
    else:
        cache = kvc.CompressedKVCache(n_slots=B, n_kv=n_kv, capacity=4112, bases=None)
        ks, vs = ([np.ascontiguousarray(O.kv_like(n_kv, max(x, 1), 7 * s + i).transpose(1, 0, 2))[:x] for s, x in enumerate(lens)] for i in (1, 2))
        for s in range(B):
            cache.prefill(s, to_bf16_cuda(ks[s]), to_bf16_cuda(vs[s]), check=False)
        call = lambda: cache.attention(to_bf16_cuda(q16), torch.arange(B, dtype=torch.int32, device="cuda"), SCALE, max_len=4100, out_f32=o32)
    for units in (19, 37, 37, 40):
        monkeypatch.setattr(kvc, "choose_units", lambda *a, u=units: u)
        monkeypatch.setattr(pk, "choose_units", lambda *a, u=units: u)
        o32.fill_(float("nan"))
        call()
        for b in range(B):
            if lens[b]:
                assert_attention_close(o32[b].cpu().numpy(), q16[b], ks[b][:lens[b]], vs[b][:lens[b]], SCALE, (b, units))
            else:
                assert not o32[b].any()


# a row whose length is negative is an empty one, as it is where every row is split alike: its output is zero and its neighbours get their ranges
@pytest.mark.gpu
@pytest.mark.parametrize("units", [4, 9, 40])
def test_negative_length_is_empty(monkeypatch, units):
    import torch
    import gaac_b200.vllm.paged_kernel as pk
    n_kv, G, lens = 2, 4, [700, 64, 33, 1500]
    st, buf, bt, ks, vs = _build_paged(lens, n_kv, 200, seed=9)
    q16 = O.f32_to_bf16((np.random.default_rng(1).standard_normal((4, n_kv * G, 128)) * 0.3).astype(np.float32))
    monkeypatch.setattr(pk, "choose_units", lambda *a: units)
    for gone in (-1, -16, -40, -(1 << 20)):
        sl = torch.tensor([700, gone, 33, 1500], dtype=torch.int32, device="cuda")
        out = torch.full((4, n_kv * G * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        o32 = torch.full((4, n_kv * G, 128), float("nan"), dtype=torch.float32, device="cuda")
        pk.paged_attention(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_kv * G, n_kv, out_f32=o32)
        assert not o32[1].any()
        for b in (0, 2, 3):
            assert_attention_close(o32[b].cpu().numpy(), q16[b], ks[b], vs[b], SCALE, (b, units, gone))
