"""Kernels that start while the one before them is still finishing: chains of calls that read what the call before wrote, queued back to back many times over, leave the same bytes as
with the overlap switched off (attention: the same up to the order of its fp32 sums)."""
import numpy as np
import pytest
from common import to_bf16_cuda
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu
N_KV, G = 4, 4


def _slots():
    import torch
    from gaac_b200 import CompressedKVCache
    k = to_bf16_cuda(O.kv_like(N_KV, 700, 1)).transpose(0, 1).contiguous()
    q, slots, out = k[:6].repeat(1, G, 1).contiguous(), torch.tensor([1, 0, 2, -1, 4, 3], dtype=torch.int32, device="cuda"), []
    cache = CompressedKVCache(5, N_KV, 1024)
    for slot, L in enumerate((500, 33, 16, 1, 640)):
        cache.prefill(slot, k[:L], k[700 - L:], check=False)
    for i in range(40):                              # every row completes blocks on the way
        cache.append(slots, k[i:i + 6], k[i + 100:i + 106])
        if i % 3 == 0: out.append(cache.attention(q, slots, 128 ** -0.5, max_len=700))
    return [t for s in (cache.k, cache.v) for t in (s.sm, s.codes, s.flags, s.tile_off, s.ovf, s.ovf_used, s.tail, s.base3, s.base4)] + [cache.S, cache.tail_len], out


def _paged(E):
    import torch
    from gaac_b200 import Codec
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    from gaac_b200.vllm.paged_kernel import paged_attention
    x = to_bf16_cuda(O.kv_like(N_KV, 16 * E + 64, 2))
    rows = x.transpose(0, 1).contiguous()
    c = Codec(N_KV).calibrate(x)
    bases = {"k3": c.base3, "k4": c.base4, "v3": c.base3, "v4": c.base4}
    blocks = 2 * E + 2
    st = LayerState(blocks, N_KV, blocks * 2 * N_KV, bases, 128, "cuda")
    buf = torch.zeros(blocks * 2 * N_KV * (OVF_OFF + 128), dtype=torch.uint8, device="cuda")
    i32 = lambda rows: torch.tensor(rows, dtype=torch.int32, device="cuda")
    # everything that a call takes is there before the first one, so that nothing but the calls' own kernels is in the stream
    freeq, rounds = torch.empty(E * 2 * N_KV, dtype=torch.int32, device="cuda"), 6
    ent = [[i32([[at + e, 16 * e + 8 * half, 8 * half, 8] for e in range(E)]) for half in (0, 1)] for at in (0, E)]
    pairs, table, lens = [i32([[at + e, 16 * e, 16] for e in range(E)]) for at in (0, E)], [i32([[at + e for e in range(E)]]) for at in (0, E)], i32([16 * E])
    back = torch.zeros(rounds, 2, 2, 16 * E, N_KV, 128, dtype=torch.bfloat16, device="cuda")
    q, out = rows[:1].repeat(1, G, 1).contiguous(), torch.zeros(rounds, 1, G * N_KV * 128, dtype=torch.bfloat16, device="cuda")
    first, flipped = rows[:16 * E].contiguous(), rows[:16 * E].flip(0).contiguous()
    # fill blocks by halves, read them back, attend over them, write over them at once with K and V exchanged, read them back; then the other end of the pool with what was read
    for r in range(rounds):
        w = r % 2
        k, v = (first, flipped) if r == 0 else back[r - 1, 1]
        for again, (a, b) in enumerate(((k, v), (v, k))):
            for half in (0, 1):
                st.store(a, b, buf, ent[w][half], freeq)
            st.decode_blocks(buf, pairs[w], back[r, again, 0], back[r, again, 1])
            if not again: paged_attention(q, out[r], buf, st.raw, st.mt, table[w], lens, st.bases, st.TS, G * N_KV, N_KV)
    return [buf, st.top, st.err, back], [out]


def _pages():
    import torch
    from gaac_b200 import Codec
    x, out = to_bf16_cuda(O.kv_like(8, 3000, 3)), []
    for i in range(6):
        c = Codec(8).calibrate(x)
        y = Codec.decode(c.encode(x, "kv"[i % 2]))
        x = y.roll(7, 1)
        out.append(y)
    return out, []


@pytest.mark.parametrize("chain", ["slots", "pages", "paged 3", "paged 60"])
def test_same_bytes(chain):
    import torch
    from gaac_b200 import _lib
    run = {"slots": _slots, "pages": _pages, "paged 3": lambda: _paged(3), "paged 60": lambda: _paged(60)}[chain]
    got = {}
    for overlap in (0, 1):
        _lib.lib().gaac_set_launch_overlap(overlap)
        try:
            got[overlap] = [run() for _ in range(3)]
            torch.cuda.synchronize()
        finally:
            _lib.lib().gaac_set_launch_overlap(1)
    for exact, near in got[0] + got[1]:
        for a, b in zip(exact, got[0][0][0]):
            assert torch.equal(a.view(torch.int16) if a.dtype == torch.bfloat16 else a, b.view(torch.int16) if b.dtype == torch.bfloat16 else b)
        for a, b in zip(near, got[0][0][1]):         # BF16 results (2^-8 between neighbours) of fp32 sums whose order varies
            assert bool(((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 1e-3).all())
