"""Merge of the splits: counts around the 32 that a warp takes at once, splits without tokens, groups of one and two sets of heads, one split; grid launches of the three kernels against
the fp64 oracle, and an infinite element, which must not reach the splits beside it."""
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu
SPLITS = [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 150]


@pytest.mark.parametrize("G", [1, 4, 5, 8])
@pytest.mark.parametrize("S", [1, 40, 1500])
def test_pages(G, S):
    import torch
    from gaac_b200 import Codec, attention
    B, n_kv = 2, 2
    k16, v16 = O.kv_like(B * n_kv, S, 1), O.kv_like(B * n_kv, S, 2)
    kp, vp = Codec(n_kv).calibrate(to_bf16_cuda(k16)).encode(to_bf16_cuda(k16), "k"), Codec(n_kv).calibrate(to_bf16_cuda(v16)).encode(to_bf16_cuda(v16), "v")
    q16 = O.f32_to_bf16((np.random.default_rng(0).standard_normal((B, n_kv * G, 128)) * 0.3).astype(np.float32))
    for nsplit in SPLITS:
        o32 = torch.empty(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
        out = attention(to_bf16_cuda(q16), kp, vp, nsplit=nsplit, out_f32=o32)
        for b in range(B):
            h = slice(b * n_kv, (b + 1) * n_kv)
            assert_attention_close(o32[b].cpu().numpy(), q16[b], k16[h].transpose(1, 0, 2), v16[h].transpose(1, 0, 2), 128 ** -0.5, nsplit)
        assert torch.equal(out, o32.to(torch.bfloat16))


@pytest.mark.parametrize("wide,G", [(False, 4), (False, 7), (True, 4), (True, 8)])
def test_paged(wide, G):
    import torch
    from gaac_b200 import Codec
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    from gaac_b200.vllm.paged_kernel import paged_attention
    from gaac_b200.vllm.paged_kernel256 import paged_attention256
    n_kv, S = 1, 700
    heads, dim = (2, 256) if wide else (1, 128)
    k16, v16 = O.kv_like(heads, S, 3), O.kv_like(heads, S, 4)
    ck, cv = Codec(heads).calibrate(to_bf16_cuda(k16)), Codec(heads).calibrate(to_bf16_cuda(v16))
    blocks = -(-S // 16)
    st = LayerState(blocks, heads, 2 * heads * blocks, {"k3": ck.base3, "k4": ck.base4, "v3": cv.base3, "v4": cv.base4}, 128, "cuda")
    buf = torch.zeros(blocks * 2 * heads * (OVF_OFF + 128), dtype=torch.uint8, device="cuda")
    kt, vt = np.ascontiguousarray(k16.transpose(1, 0, 2)), np.ascontiguousarray(v16.transpose(1, 0, 2))
    ent = torch.tensor([[b, 16 * b, 0, min(16, S - 16 * b)] for b in range(blocks)], dtype=torch.int32, device="cuda")
    st.store(to_bf16_cuda(kt), to_bf16_cuda(vt), buf, ent, torch.empty(blocks * 2 * heads, dtype=torch.int32, device="cuda"))
    q16 = O.f32_to_bf16((np.random.default_rng(0).standard_normal((1, G, dim)) * 0.3).astype(np.float32))
    bt, sl = torch.arange(blocks, dtype=torch.int32, device="cuda")[None], torch.tensor([S], dtype=torch.int32, device="cuda")
    for nsplit in SPLITS:
        out, o32 = torch.empty(1, G * dim, dtype=torch.bfloat16, device="cuda"), torch.empty(1, G, dim, dtype=torch.float32, device="cuda")
        (paged_attention256 if wide else paged_attention)(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, G, n_kv, nsplit, out_f32=o32)
        assert_attention_close(o32[0].cpu().numpy(), q16[0], kt.reshape(S, n_kv, dim), vt.reshape(S, n_kv, dim), dim ** -0.5, nsplit)


def test_infinite_element_in_the_last_split():
    import torch
    from gaac_b200 import Codec, attention
    S, G = 700, 4
    k16, v16 = O.kv_like(1, S, 1, outliers=0.0), O.kv_like(1, S, 2, outliers=0.0)
    v16[0, S - 1, 5] = 0x7F80
    kp, vp = Codec(1).calibrate(to_bf16_cuda(k16)).encode(to_bf16_cuda(k16), "k"), Codec(1).calibrate(to_bf16_cuda(v16)).encode(to_bf16_cuda(v16), "v")
    q = to_bf16_cuda(O.f32_to_bf16((np.random.default_rng(0).standard_normal((1, G, 128)) * 0.1).astype(np.float32)))
    for nsplit in SPLITS:
        out = attention(q, kp, vp, nsplit=nsplit).float()
        assert bool(torch.isinf(out[..., 5]).all()) and bool(torch.isfinite(out[..., :5]).all()) and bool(torch.isfinite(out[..., 6:]).all()), nsplit
