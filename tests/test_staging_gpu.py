"""Attention over escape-heavy tiles, around what a stage has room for: no group promoted, some, every group (256 escape bytes), every group and some raw
ones, every group raw (1280), and tiles of both kinds side by side; read from staged bytes or from global memory, against the fp64 oracle."""
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


def _tables(x16, heads, mode):
    """Base tables that make groups of x16 [heads, S, 128] fall out of the 3-bit window (base 0) or out of both."""
    b3, b4 = O.calibrate(x16, heads)
    ch = np.arange(128)
    miss3 = {"none": ch < 0, "half": ch % 16 < 2, "all": ch >= 0, "raw": ch >= 0, "some raw": ch >= 0}[mode]
    miss4 = {"raw": ch >= 0, "some raw": ch == 5}.get(mode, ch < 0)
    b3[:, miss3] = 0
    b4[:, miss4] = 0
    return b3, b4


def _data(heads, S, seed, mixed):
    x = O.synth_kv("v", heads, S, seed, raw_frac=0.0, four_frac=0.0)
    if mixed:                                        # every fifth tile of random exponents: all of its groups raw, 1280 escape bytes
        e = np.random.default_rng(seed).integers(90, 134, x.shape).astype(np.uint16)
        t = (np.arange(S) // 16 % 5 == 2)[None, :, None]
        x = np.where(t, (x & 0x807F) | (e << 7), x)
    return np.ascontiguousarray(x)


@pytest.mark.parametrize("mode", ["none", "half", "all", "some raw", "raw"])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n_kv,G", [(2, 4), (1, 8)])
def test_pages(mode, mixed, n_kv, G):
    import torch
    from gaac_b200 import Codec, attention
    S = 1333
    k16, v16 = _data(n_kv, S, 1, mixed), _data(n_kv, S, 2, mixed)
    pg = []
    for kind, x in (("k", k16), ("v", v16)):
        b3, b4 = _tables(x, n_kv, mode)
        pg.append(Codec(n_kv).set_bases(torch.from_numpy(b3), torch.from_numpy(b4)).encode(to_bf16_cuda(x), kind))
    q16 = O.f32_to_bf16((np.random.default_rng(0).standard_normal((1, n_kv * G, 128)) * 0.3).astype(np.float32))
    for nsplit in (1, 3):
        o32 = torch.empty(1, n_kv * G, 128, dtype=torch.float32, device="cuda")
        attention(to_bf16_cuda(q16), *pg, nsplit=nsplit, out_f32=o32)
        assert_attention_close(o32[0].cpu().numpy(), q16[0], k16.transpose(1, 0, 2), v16.transpose(1, 0, 2), 128 ** -0.5, nsplit)


@pytest.mark.parametrize("mode", ["none", "half", "all", "some raw", "raw"])
@pytest.mark.parametrize("ovf_slot", [128, 144, 240, 256, 272, 1280])
@pytest.mark.parametrize("wide,n_kv,G", [(False, 2, 4), (False, 1, 8), (True, 1, 4), (True, 1, 7)])
def test_paged(mode, ovf_slot, wide, n_kv, G):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    from gaac_b200.vllm.paged_kernel import paged_attention
    from gaac_b200.vllm.paged_kernel256 import paged_attention256
    heads, dim, S = (2 * n_kv, 256, 905) if wide else (n_kv, 128, 905)
    k16, v16, bases = _data(heads, S, 3, True), _data(heads, S, 4, True), {}
    for kind, x in (("k", k16), ("v", v16)):
        bases[kind + "3"], bases[kind + "4"] = (torch.from_numpy(b) for b in _tables(x, heads, mode))
    blocks = -(-S // 16)
    st = LayerState(blocks, heads, raw_tiles=2 * heads * blocks, bases=bases, ovf_slot=ovf_slot, device="cuda")
    buf = torch.zeros(blocks * 2 * heads * (OVF_OFF + ovf_slot), dtype=torch.uint8, device="cuda")
    kt, vt = np.ascontiguousarray(k16.transpose(1, 0, 2)), np.ascontiguousarray(v16.transpose(1, 0, 2))
    ent = torch.tensor([[b, 16 * b, 0, min(16, S - 16 * b)] for b in range(blocks)], dtype=torch.int32, device="cuda")
    st.store(to_bf16_cuda(kt), to_bf16_cuda(vt), buf, ent, torch.empty(blocks * 2 * heads, dtype=torch.int32, device="cuda"))
    n_q = n_kv * G
    q16 = O.f32_to_bf16((np.random.default_rng(0).standard_normal((1, n_q, dim)) * 0.3).astype(np.float32))
    bt, sl = torch.arange(blocks, dtype=torch.int32, device="cuda")[None], torch.tensor([S], dtype=torch.int32, device="cuda")
    out, o32 = torch.empty(1, n_q * dim, dtype=torch.bfloat16, device="cuda"), torch.empty(1, n_q, dim, dtype=torch.float32, device="cuda")
    (paged_attention256 if wide else paged_attention)(to_bf16_cuda(q16), out, buf, st.raw, st.mt, bt, sl, st.bases, st.TS, n_q, n_kv, 2, out_f32=o32)
    assert_attention_close(o32[0].cpu().numpy(), q16[0], kt.reshape(S, n_kv, dim), vt.reshape(S, n_kv, dim), dim ** -0.5, ovf_slot)
