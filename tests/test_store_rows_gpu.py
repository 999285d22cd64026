"""Rows of a store step, in one or two steps per block: the new rows of a block that fills travel ahead of the mode-table entry, its old ones and those of a part of a block behind it; a block that
fills is gathered from both; one whose escape bytes do not fit its slot stays raw.  What comes back out of the blocks is what went in, bit for bit, on both sides of the
store's two forms (one cluster, two launches)."""
import numpy as np
import pytest
from common import to_bf16_cuda, bits
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu
N_KV, OVF_SLOT = 2, 128


@pytest.mark.parametrize("E", [3, 30])                         # 12 and 120 tiles
@pytest.mark.parametrize("noise", [False, True])               # fits its slot when full; does not
@pytest.mark.parametrize("off0,n", [(0, 1), (0, 2), (0, 3), (0, 15), (0, 16), (1, 1), (5, 2), (5, 3), (5, 11), (13, 3), (15, 1)])
def test_rows_come_back(E, noise, off0, n):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    rng = np.random.default_rng(100 * off0 + n)
    shape = (E * 16, N_KV, 128)
    if noise: k, v = (rng.integers(0, 1 << 16, shape).astype(np.uint16) for _ in range(2))
    else: k, v = (np.ascontiguousarray(O.synth_kv(c, N_KV, E * 16, 7).transpose(1, 0, 2)) for c in "kv")
    k3, k4 = O.calibrate(O.synth_kv("k", N_KV, 2048, 7), N_KV); v3, v4 = O.calibrate(O.synth_kv("v", N_KV, 2048, 7), N_KV)
    st = LayerState(2 * E, N_KV, 2 * N_KV * E, {a: torch.from_numpy(b) for a, b in (("k3", k3), ("k4", k4), ("v3", v3), ("v4", v4))}, OVF_SLOT, "cuda")
    buf = torch.zeros(2 * E * 2 * N_KV * (OVF_OFF + OVF_SLOT), dtype=torch.uint8, device="cuda")
    kd, vd = to_bf16_cuda(k), to_bf16_cuda(v)
    blocks = rng.permutation(2 * E)[:E]
    freeq = torch.empty(E * 2 * N_KV, dtype=torch.int32, device="cuda")
    for first, count in ((0, off0), (off0, n)):
        if count: st.store(kd, vd, buf, torch.tensor([[b, 16 * i + first, first, count] for i, b in enumerate(blocks)], dtype=torch.int32, device="cuda"), freeq)
    sk = torch.zeros(E * 16, N_KV, 128, dtype=torch.bfloat16, device="cuda"); sv = torch.zeros_like(sk)
    st.decode_blocks(buf, torch.tensor([[b, 16 * i, off0 + n] for i, b in enumerate(blocks)], dtype=torch.int32, device="cuda"), sk, sv)
    rows = (np.arange(E * 16) % 16) < off0 + n
    assert np.array_equal(bits(sk)[rows], k[rows]) and np.array_equal(bits(sv)[rows], v[rows])
    assert not bits(sk)[~rows].any() and not bits(sv)[~rows].any()                             # (rows that the block does not have are not written)
    raw = (st.mt.cpu().numpy() < 0).sum()
    assert raw == (0 if off0 + n == 16 and not noise else 2 * N_KV * E) and int(st.top) == 2 * N_KV * E - raw and int(st.err) == 0
