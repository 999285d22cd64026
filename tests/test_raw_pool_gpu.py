"""A raw pool that runs empty: the blocks that got no tile lose their rows and nothing else happens - no other block's rows, nothing outside the stack, no
tile that is handed out twice - for steps that the store takes in one launch and in two."""
import numpy as np
import pytest
from common import to_bf16_cuda, bits
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 4, 11, 12, 44, 45, 60])    # 2 * E tile slots; up to 88 are one launch, of 11 per block
@pytest.mark.parametrize("short", [1, 2])
@pytest.mark.parametrize("end", ["fill", "release"])
def test_pool_runs_empty(E, short, end):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    R, none = 2 * E - short, ~(1 << 30)
    if R == 0:
        pytest.skip("a pool of no tiles")
    k16, v16 = (O.synth_kv(kind, 1, 16 * E, E, raw_frac=0.0, four_frac=0.05).transpose(1, 0, 2) for kind in "kv")
    bases = {}
    for kind, x16 in (("k", k16), ("v", v16)):
        bases[kind + "3"], bases[kind + "4"] = (torch.from_numpy(b) for b in O.calibrate(np.ascontiguousarray(x16.transpose(1, 0, 2)), 1))
    st = LayerState(E, 1, raw_tiles=R, bases=bases, ovf_slot=1280, device="cuda")
    guarded = torch.full((R + 16,), -7, dtype=torch.int32, device="cuda")
    st.stack = guarded[8:8 + R].copy_(st.stack)
    buf = torch.zeros(E * 2 * (OVF_OFF + 1280), dtype=torch.uint8, device="cuda")
    k, v = to_bf16_cuda(k16), to_bf16_cuda(v16)
    freeq = torch.empty(2 * E, dtype=torch.int32, device="cuda")

    def step(off, n):
        st.store(k, v, buf, torch.tensor([[b, 16 * b + off, off, n] for b in range(E)], dtype=torch.int32, device="cuda"), freeq)

    def rows(n):                                     # [E, 2 (kind)]: the block's first n rows read back as they were stored
        sk = torch.zeros(16 * E, 1, 128, dtype=torch.bfloat16, device="cuda"); sv = torch.zeros_like(sk)
        st.decode_blocks(buf, torch.tensor([[b, 16 * b, n] for b in range(E)], dtype=torch.int32, device="cuda"), sk, sv)
        return np.stack([(bits(got).reshape(E, 16, 128)[:, :n] == want.reshape(E, 16, 128)[:, :n]).all((1, 2)) for got, want in ((sk, k16), (sv, v16))], 1)

    step(0, 9)
    dud = (st.mt.view(E, 2) == none).cpu().numpy()
    assert int(st.err) == short == dud.sum() and int(st.top) <= 0
    assert np.array_equal(rows(9), ~dud)
    step(9, 6)                                       # the blocks without a tile ask again, in vain
    assert int(st.err) == 2 * short and np.array_equal((st.mt.view(E, 2) == none).cpu().numpy(), dud) and np.array_equal(rows(15), ~dud)
    if end == "fill":                                # every block compresses (the slots have room for any tile); what was never popped does not come back
        step(15, 1)
        assert (st.mt >= 0).all() and np.array_equal(rows(16), ~dud)
    else:
        st.release_blocks(torch.arange(E, dtype=torch.int32, device="cuda"))
    assert int(st.top) == R and sorted(st.stack.tolist()) == list(range(R)) and torch.equal(st.mt, torch.arange(2 * E, dtype=torch.int32, device="cuda"))
    assert (guarded[:8] == -7).all() and (guarded[8 + R:] == -7).all()
    st.release_blocks(torch.arange(E, dtype=torch.int32, device="cuda"))          # nothing left to release
    assert int(st.top) == R
    errs = int(st.err)
    st.store(k, v, buf, torch.tensor([[0, 0, 0, 3]], dtype=torch.int32, device="cuda"), freeq)                    # the pool serves again
    assert int(st.err) == errs + (R < 2) and (st.mt.view(E, 2)[0] < 0).all() and rows(3)[0].sum() == min(2, R)
