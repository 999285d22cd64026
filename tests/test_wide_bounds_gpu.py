"""Grids whose split count was chosen for rows far longer than those that there are: rows of few tiles take fewer ranges (fewer_ranges in gaac_attn.cu), the CTAs that get none
leave.  Rows around one tile per warp (16, at head_dim 256 eight), around four tiles per range, empty ones and ones that are all tail, against the fp64 oracle; infinite elements, which
are summed by a pass of its own over the same ranges; and the rules that choose such grids."""
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O
from test_paged_gpu import _build_paged

SCALE = 128 ** -0.5
LENS = [1, 16, 127, 129, 255, 256, 257, 273, 700, 1030]


def test_rules():
    from gaac_b200.kernel import choose_nsplit256, choose_nsplit_sm100, choose_units
    for n_kv in (1, 2, 4, 8, 148, 149):
        for B in (1, 2, 5, 9, 32, 64, 200):
            for S in (0, 1, 16, 272, 273, 1000, 5000, 10 ** 6):
                rows, ns, ns256 = B * n_kv, choose_nsplit_sm100(B, n_kv, S, ragged=True), choose_nsplit256(B, n_kv, S)
                assert ns >= 1 and ns256 >= 1
                if 1 < B <= rows <= 148 and -(-S // 16) <= 17 * (148 // rows):
                    assert choose_units(B, n_kv, S) == 0 and rows * ns <= 148                  # one wave
    assert choose_units(2, 8, 2000) == 0 and choose_nsplit_sm100(2, 8, 2000, ragged=True) == 9 and choose_units(2, 8, 8000) == 18
    assert choose_nsplit256(8, 4, 500) == 4 and choose_nsplit256(1, 1, 64) == 1


def _slots(lens, n_kv, change=None, **gen):
    import gaac_b200.kv_cache as kvc
    cache, hist = kvc.CompressedKVCache(n_slots=len(lens), n_kv=n_kv, capacity=2048, bases=None), []
    for s, L in enumerate(lens):
        k, v = (np.ascontiguousarray(O.kv_like(n_kv, max(L, 1), 7 * s + i, **gen).transpose(1, 0, 2))[:L] for i in (1, 2))
        if change: change(s, k, v)
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v), check=False)
        hist.append((k, v))
    return cache, hist


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G", [(2, 4), (1, 8)])
def test_slots(n_kv, G):
    import torch
    lens = LENS + [0, 3]
    cache, hist = _slots(lens, n_kv)
    q16 = O.f32_to_bf16((np.random.default_rng(G).standard_normal((len(lens), n_kv * G, 128)) * 0.1).astype(np.float32))
    o32 = torch.empty(len(lens), n_kv * G, 128, dtype=torch.float32, device="cuda")
    for nsplit in (1, 2, 5, 16, 74, 74):              # the same call twice: the split counters are left at zero
        o32.fill_(float("nan"))
        cache.attention(to_bf16_cuda(q16), torch.arange(len(lens), dtype=torch.int32, device="cuda"), SCALE, nsplit=nsplit, out_f32=o32)
        for b, L in enumerate(lens):
            if L == 0: assert not o32[b].any()
            else: assert_attention_close(o32[b].cpu().numpy(), q16[b], *hist[b], SCALE, (L, nsplit))


@pytest.mark.gpu
def test_slots_with_infinite_elements():
    """An infinite element of V reaches its own channel only, whatever range it lies in."""
    import torch
    lens, at = [257, 700, 40], [200, 650, 3]
    def change(s, k, v): v[at[s], 0, 5 + s] = 0x7F80
    cache, hist = _slots(lens, 1, change, outliers=0.0)                             # (no weight underflows: 0 x Inf is NaN)
    q16 = O.f32_to_bf16((np.random.default_rng(2).standard_normal((3, 4, 128)) * 0.1).astype(np.float32))
    o32 = torch.empty(3, 4, 128, dtype=torch.float32, device="cuda")
    for nsplit in (3, 40):
        cache.attention(to_bf16_cuda(q16), torch.arange(3, dtype=torch.int32, device="cuda"), SCALE, nsplit=nsplit, out_f32=o32)
        for b in range(3):
            o, (k, v) = o32[b].cpu().numpy().copy(), hist[b]
            assert (o[:, 5 + b] == np.inf).all()
            v = v.copy(); v[at[b], 0, 5 + b] = 0
            ref = O.attention_ref(q16[b], k, v, SCALE)
            o[:, 5 + b] = ref[:, 5 + b]
            assert_attention_close(o, q16[b], k, v, SCALE, (b, nsplit))


@pytest.mark.gpu
@pytest.mark.parametrize("n_kv,G,wide", [(2, 4, False), (1, 8, False), (1, 4, True), (2, 6, True)])
def test_paged(n_kv, G, wide):
    import torch
    from gaac_b200.vllm.paged_kernel import paged_attention
    from gaac_b200.vllm.paged_kernel256 import paged_attention256
    dim, halves = (256, 2) if wide else (128, 1)
    st, buf, bt, ks, vs = _build_paged(LENS, halves * n_kv, sum(-(-x // 16) for x in LENS) + 4, seed=n_kv + G, adversarial_every=5, raw_tiles=halves * 2 * n_kv * 256)
    bt = torch.nn.functional.pad(bt, (0, 512 - bt.shape[1])).contiguous()                  # a table of 8192 tokens
    q16 = O.f32_to_bf16((np.random.default_rng(1).standard_normal((len(LENS), n_kv * G, dim)) * 0.3).astype(np.float32))
    sl = torch.tensor(LENS, dtype=torch.int32, device="cuda")
    out = torch.empty(len(LENS), n_kv * G * dim, dtype=torch.bfloat16, device="cuda")
    o32 = torch.empty(len(LENS), n_kv * G, dim, dtype=torch.float32, device="cuda")
    for nsplit in (1, 2, 7, 14, 74, 74, None):
        o32.fill_(float("nan"))
        (paged_attention256 if wide else paged_attention)(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_kv * G, n_kv, nsplit=nsplit, out_f32=o32)
        for b, L in enumerate(LENS):
            k, v = ks[b].reshape(L, n_kv, dim), vs[b].reshape(L, n_kv, dim)
            assert_attention_close(o32[b].cpu().numpy(), q16[b], k, v, dim ** -0.5, (L, nsplit))
