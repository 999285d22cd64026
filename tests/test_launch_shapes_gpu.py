"""Encode and decode at the sizes where a launch changes its shape (one, two, three, four tiles per warp), with CTAs that are not full: every head's bytes are those of the
same head encoded in a batch of a few heads, where a warp has one tile; a few heads against the oracle."""
import numpy as np
import pytest
from common import to_bf16_cuda, bits
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [369, 370, 555, 592, 740])              # 14 tiles: 4 CTAs of one tile per warp and head;  740 and 1184 of them are one wave
@pytest.mark.parametrize("kind", ["k", "v"])
def test_tiles_per_warp(H, kind):
    import torch
    from gaac_b200 import Codec
    S, few, n_kv = 13 * 16 + 5, 5, 2
    base = O.kv_like(few * n_kv, S, seed=3)
    x = to_bf16_cuda(np.ascontiguousarray(np.resize(base, (H, S, 128))))
    codec = Codec(n_kv).calibrate(to_bf16_cuda(base))
    small, big = codec.encode(to_bf16_cuda(base), kind), codec.encode(x, kind)
    h = torch.arange(H, device="cuda") % (few * n_kv)
    for f in ("sm", "codes", "flags", "tile_off"):
        assert torch.equal(getattr(big, f), getattr(small, f)[h]), f
    size = (small.ovf_head_start[1:] - small.ovf_head_start[:-1])[h]
    assert torch.equal(big.ovf_head_start[1:], size.cumsum(0).int())
    a, b = big.ovf_head_start.tolist(), small.ovf_head_start.tolist()
    for i in {0, 1, few * n_kv, H // 2, H - 2, H - 1}:
        j = i % (few * n_kv)
        assert torch.equal(big.ovf[a[i]:a[i + 1]], small.ovf[b[j]:b[j + 1]]), i
    rel = big.ovf_off - big.ovf_off[:, :1]
    assert torch.equal(rel, small.ovf_off[h] - small.ovf_off[h][:, :1])
    assert np.array_equal(bits(Codec.decode(big)), bits(x))
    ref = O.encode(base, codec.base3.cpu().numpy(), codec.base4.cpu().numpy(), kind, n_kv)
    assert np.array_equal(small.sm.cpu().numpy(), ref["sm"]) and np.array_equal(small.flags.cpu().numpy(), ref["flags"])
