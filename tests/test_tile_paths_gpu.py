"""Edges of the encoder, the decoder, the calibration and the prefill: sizes around their tiles, chunks and thresholds, escape-heavy tiles, slots that
are not 32-byte aligned.  Everything is bit-exact against the oracle."""
import numpy as np
import pytest
from common import to_bf16_cuda, bits, page_to_dict, assert_pages_equal
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


# heads: around the 64 up to which one warp makes the prefix over the heads, and past the block's 1024; tokens: around a tile, the 16 tiles of a copy
# block and of an encode block; random bits: tiles with more escape bytes (up to 1280) than the decoder stages
@pytest.mark.parametrize("kind", ["k", "v"])
@pytest.mark.parametrize("H,S,random_bits", [(1, 1, False), (2, 15, False), (3, 17, True), (64, 33, False), (65, 257, True), (2, 4177, False), (1030, 16, False)])
def test_encode_decode_edges(kind, H, S, random_bits):
    import torch
    from gaac_b200 import Codec
    n_kv = 2 if H % 2 == 0 else 1
    rng = np.random.default_rng(H * 1000 + S)
    x16 = rng.integers(0, 65536, (H, S, 128)).astype(np.uint16) if random_bits else O.synth_kv(kind, H, S, S, raw_frac=0.03, four_frac=0.2)
    b3, b4 = O.calibrate(O.synth_kv(kind, n_kv, 256, S), n_kv)
    codec = Codec(n_kv).set_bases(torch.from_numpy(b3), torch.from_numpy(b4))
    x = to_bf16_cuda(x16)
    pg = codec.encode(x, kind)
    assert_pages_equal(page_to_dict(pg), O.encode(x16, b3, b4, kind, n_kv))
    assert torch.equal(Codec.decode(pg).view(torch.int16), x.view(torch.int16))


# the smallest and largest base tables that leave room for their windows, and exponents on both sides of every window's ends
@pytest.mark.parametrize("kind", ["k", "v"])
@pytest.mark.parametrize("b3v,b4v", [(0, 0), (248, 240), (100, 96), (7, 239)])
def test_windows_at_the_ends_of_the_exponent_range(kind, b3v, b4v):
    import torch
    from gaac_b200 import Codec
    rng = np.random.default_rng(b3v)
    near = np.array([b3v - 1, b3v, b3v + 7, b3v + 8, b4v - 1, b4v, b4v + 15, b4v + 16, 0, 255]).clip(0, 255)
    near = np.concatenate([near, np.arange(b3v, b3v + 8).repeat(40), np.arange(b4v, b4v + 16).repeat(4)])
    e = rng.choice(near, (2, 64, 128)).astype(np.uint16)
    x16 = ((e << 7) | rng.integers(0, 128, e.shape).astype(np.uint16) | (rng.integers(0, 2, e.shape).astype(np.uint16) << 15)).astype(np.uint16)
    b3, b4 = np.full((2, 128), b3v, np.uint8), np.full((2, 128), b4v, np.uint8)
    pg = Codec(2).set_bases(torch.from_numpy(b3), torch.from_numpy(b4)).encode(to_bf16_cuda(x16), kind)
    assert_pages_equal(page_to_dict(pg), O.encode(x16, b3, b4, kind, 2))
    assert np.array_equal(bits(Codec.decode(pg)), x16)


# rows per block (128), the unrolled part (64 rows of it) and their remainders; one exponent only: a counter reaches the block's 128
@pytest.mark.parametrize("N", [1, 3, 63, 64, 65, 127, 128, 129, 333])
@pytest.mark.parametrize("constant", [False, True])
def test_histogram_edges(N, constant):
    import torch
    from gaac_b200.codec import exponent_hist
    x16 = np.full((N, 3, 128), 0x3F80, np.uint16) if constant else np.random.default_rng(N).integers(0, 65536, (N, 3, 128)).astype(np.uint16)
    got = exponent_hist(to_bf16_cuda(x16), 3).cpu().numpy()
    e = ((x16 >> 7) & 0xFF).reshape(N, 384)
    ref = np.stack([np.bincount(e[:, c], minlength=256) for c in range(384)])
    assert np.array_equal(got, ref)


# prompts calibrated on themselves: no whole tile, every tail length's ends, K and V rows of different strides
@pytest.mark.parametrize("L", [0, 1, 15, 16, 31, 300])
@pytest.mark.parametrize("strided", [False, True])
def test_prefill_edges(L, strided):
    import torch
    from gaac_b200 import CompressedKVCache
    n_kv = 3
    k16, v16 = O.synth_kv("k", n_kv, max(L, 1), L + 1).transpose(1, 0, 2)[:L], O.synth_kv("v", n_kv, max(L, 1), L + 1).transpose(1, 0, 2)[:L]
    k, v = to_bf16_cuda(k16), to_bf16_cuda(v16)
    if strided:
        wide = torch.zeros(max(L, 1), n_kv + 2, 128, dtype=torch.bfloat16, device="cuda")[:L]
        wide[:, :n_kv] = k
        k = wide[:, :n_kv]
    cache = CompressedKVCache(n_slots=2, n_kv=n_kv, capacity=320, bases=None)
    cache.prefill(1, k, v)
    if L:
        gk, gv = cache.decompress(1)
        assert np.array_equal(bits(gk), k16) and np.array_equal(bits(gv), v16)
        b3, b4 = O.calibrate(np.ascontiguousarray(v16.transpose(1, 0, 2)), n_kv)
        assert np.array_equal(cache.v.base3[n_kv:].cpu().numpy(), b3) and np.array_equal(cache.v.base4[n_kv:].cpu().numpy(), b4)
    assert cache.S[n_kv:].tolist() == [L // 16 * 16] * n_kv and cache.tail_len[n_kv:].tolist() == [L % 16] * n_kv
    assert cache._slot_status[1].tolist() == [0, int(cache.k.ovf_used[n_kv:].max()), 0, int(cache.v.ovf_used[n_kv:].max())]
    assert not cache.S[:n_kv].any() and not cache.tail_len[:n_kv].any()               # the other slot is untouched


# slots of an odd multiple of 16 bytes: every second one is not 32-byte aligned; more escape bytes than the decoder stages (ovf_slot 528)
@pytest.mark.parametrize("ovf_slot", [16, 48, 128, 528])
def test_paged_slots_of_any_alignment(ovf_slot):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    n_kv, blocks = 2, 5
    k16, v16 = (O.synth_kv(kind, n_kv, 16 * blocks, 5, raw_frac=0.2 if ovf_slot > 128 else 0.0, four_frac=0.05 if ovf_slot > 16 else 0.0).transpose(1, 0, 2) for kind in "kv")
    bases = {}
    for kind, x16 in (("k", k16), ("v", v16)):
        bases[kind + "3"], bases[kind + "4"] = (torch.from_numpy(b) for b in O.calibrate(np.ascontiguousarray(x16.transpose(1, 0, 2)), n_kv))
    st = LayerState(blocks, n_kv, raw_tiles=2 * n_kv * blocks, bases=bases, ovf_slot=ovf_slot, device="cuda")
    buf = torch.zeros(blocks * 2 * n_kv * (OVF_OFF + ovf_slot), dtype=torch.uint8, device="cuda")
    ent = torch.tensor([[b, 16 * b, 0, 16] for b in range(blocks)], dtype=torch.int32, device="cuda")
    st.store(to_bf16_cuda(k16), to_bf16_cuda(v16), buf, ent, torch.empty(blocks * 2 * n_kv, dtype=torch.int32, device="cuda"))
    pairs = torch.tensor([[b, 16 * b, 16 if b else 9] for b in range(blocks)], dtype=torch.int32, device="cuda")
    sk = torch.zeros(16 * blocks, n_kv, 128, dtype=torch.bfloat16, device="cuda"); sv = torch.zeros_like(sk)
    st.decode_blocks(buf, pairs, sk, sv)
    rows = np.r_[0:9, 16:16 * blocks]
    assert np.array_equal(bits(sk)[rows], k16[rows]) and np.array_equal(bits(sv)[rows], v16[rows]) and not sk[9:16].any()
    assert int((st.mt >= 0).sum()) > 0                 # some tiles are compressed


# a step's tile slots around what one block and one cluster of the store take (10 and 80): raw tiles are popped, then all returned when the blocks fill
@pytest.mark.parametrize("E", [1, 5, 6, 10, 11, 20, 21, 40, 41])
def test_paged_store_steps_pop_and_return_raw_tiles(E):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    k16, v16 = (O.synth_kv(kind, 1, 16 * E, E, raw_frac=0.0, four_frac=0.05).transpose(1, 0, 2) for kind in "kv")
    bases = {}
    for kind, x16 in (("k", k16), ("v", v16)):
        bases[kind + "3"], bases[kind + "4"] = (torch.from_numpy(b) for b in O.calibrate(np.ascontiguousarray(x16.transpose(1, 0, 2)), 1))
    st = LayerState(E + 1, 1, raw_tiles=2 * E + 3, bases=bases, ovf_slot=512, device="cuda")
    buf = torch.zeros((E + 1) * 2 * (OVF_OFF + 512), dtype=torch.uint8, device="cuda")
    k, v = to_bf16_cuda(k16), to_bf16_cuda(v16)
    freeq = torch.empty((E + 1) * 2, dtype=torch.int32, device="cuda")
    for off, n in ((0, 15), (15, 1)):
        ent = torch.tensor([[b + 1 if b < E else -1, 16 * b + off, off, n] for b in range(E + (E % 5 == 1))], dtype=torch.int32, device="cuda")      # sometimes with an inactive entry
        st.store(k, v, buf, ent, freeq)
        assert int(st.top) == (3 if off == 0 else 2 * E + 3) and int(st.err) == 0
    assert sorted(st.stack.tolist()) == list(range(2 * E + 3)) and (st.mt >= 0).all()
    sk = torch.zeros(16 * E, 1, 128, dtype=torch.bfloat16, device="cuda"); sv = torch.zeros_like(sk)
    st.decode_blocks(buf, torch.tensor([[b + 1, 16 * b, 16] for b in range(E)], dtype=torch.int32, device="cuda"), sk, sv)
    assert np.array_equal(bits(sk), k16) and np.array_equal(bits(sv), v16)
