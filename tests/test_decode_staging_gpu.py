"""The decoders stage all of a tile's escape bytes: tiles without any, with a few, around the words that travel with the tile (128 bytes), with every group promoted, with every group raw; the block
decoder for slots whose escape room is smaller than any of that."""
import numpy as np
import pytest
from common import to_bf16_cuda, bits
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


def _tiles(kind, n_kv, tiles, seed):
    """Tiles of growing numbers of escape bytes: promoted groups only, raw ones only, both."""
    x = O.synth_kv(kind, n_kv, 16 * tiles, seed, raw_frac=0.0, four_frac=0.0)
    rng = np.random.default_rng(seed)
    for t in range(tiles):
        share = [0.0, 0.02, 0.45, 0.55, 1.0][t % 5]
        noise = rng.integers(0, 65536, x[:, 16 * t:16 * t + 16].shape).astype(np.uint16)
        near = x[:, 16 * t:16 * t + 16] + (np.uint16(4) << 7)                  # exponents four up: often beyond the 3-bit window
        hit = rng.random(noise.shape) < share / (8 if t % 3 else 1)
        x[:, 16 * t:16 * t + 16] = np.where(hit, near if t % 2 else noise, x[:, 16 * t:16 * t + 16])
    return x


@pytest.mark.parametrize("kind", ["k", "v"])
@pytest.mark.parametrize("S_off", [0, 5])
def test_pages(kind, S_off):
    from gaac_b200 import Codec
    x = np.ascontiguousarray(_tiles(kind, 3, 15, 7)[:, :240 - S_off])
    codec = Codec(3).calibrate(to_bf16_cuda(O.synth_kv(kind, 3, 512, 7)))
    pg = codec.encode(to_bf16_cuda(x), kind)
    sizes = np.diff(np.append(pg.tile_off.cpu().numpy()[0], int(pg.ovf_head_start[1])))
    assert sizes.max() > 1000 and (sizes < 128).any() and ((sizes > 128) & (sizes < 1000)).any()
    assert np.array_equal(bits(Codec.decode(pg)), x)


@pytest.mark.parametrize("ovf_slot", [0, 16, 64, 128, 256, 1280])
def test_blocks(ovf_slot):
    import torch
    from gaac_b200.vllm.store import LayerState, OVF_OFF
    n_kv, tiles = 2, 15
    ks, vs = (np.ascontiguousarray(_tiles(kind, n_kv, tiles, 11 + i).transpose(1, 0, 2)) for i, kind in enumerate("kv"))
    bases = {}
    for kind, x in (("k", ks), ("v", vs)):
        b3, b4 = O.calibrate(O.synth_kv(kind, n_kv, 512, 11 if kind == "k" else 12), n_kv)
        bases[kind + "3"], bases[kind + "4"] = torch.from_numpy(b3), torch.from_numpy(b4)
    st = LayerState(tiles, n_kv, raw_tiles=2 * tiles * n_kv, bases=bases, ovf_slot=ovf_slot, device="cuda")
    buf = torch.zeros(tiles * 2 * n_kv * (OVF_OFF + ovf_slot), dtype=torch.uint8, device="cuda")
    L = 16 * tiles - 3
    ent = torch.tensor([[t, 16 * t, 0, min(16, L - 16 * t)] for t in range(tiles)], dtype=torch.int32, device="cuda")
    st.store(to_bf16_cuda(ks[:L]), to_bf16_cuda(vs[:L]), buf, ent, torch.empty(tiles * 2 * n_kv, dtype=torch.int32, device="cuda"))
    assert int(st.err) == 0
    compressed = int((st.mt >= 0).sum())
    assert (compressed > 0 or ovf_slot < 64) and (ovf_slot == 1280 or compressed < 2 * n_kv * (tiles - 1))
    sk, sv = (torch.zeros(16 * tiles, n_kv, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    st.decode_blocks(buf, torch.tensor([[t, 16 * t, min(16, L - 16 * t)] for t in range(tiles)], dtype=torch.int32, device="cuda"), sk, sv)
    assert np.array_equal(bits(sk)[:L], ks[:L]) and np.array_equal(bits(sv)[:L], vs[:L])
    assert not bits(sk)[L:].any() and not bits(sv)[L:].any()
