"""Short ranges as clusters whose partials meet in shared memory (teams): every number of ranges up to eight and one beyond, ranges as long as a team takes them (24 tiles) and longer, rows with fewer ranges
than CTAs, more rows than the GPU has room for, groups of 1 to 8; against the fp64 oracle, and the same call twice."""
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O

SCALE = 128 ** -0.5


def test_rules():
    from gaac_b200.kernel import TEAMS, _team, choose_nsplit_sm100
    assert [_team(r) for r in (1, 15, 16, 22, 26, 33, 45, 74, 75)] == [8, 8, 6, 6, 5, 4, 3, 2, 1]
    assert all(n * TEAMS[n] <= 148 for n in TEAMS)
    assert choose_nsplit_sm100(1, 8, 128) == 1 and choose_nsplit_sm100(1, 8, 500) == 8 and choose_nsplit_sm100(2, 8, 1000) == 6 and choose_nsplit_sm100(1, 8, 2000) == 16


@pytest.mark.gpu
def test_the_gpu_has_the_room_that_the_rules_count_on():
    """Otherwise the launches of this file would pass as grids."""
    import torch
    from gaac_b200 import _lib
    from gaac_b200.kernel import TEAMS
    room = _lib.lib().gaac_debug_team_room
    assert torch.cuda.get_device_properties(0).multi_processor_count != 148 or all(room(paged, G, n) >= TEAMS[n] for paged in (0, 1) for G in (1, 4, 5, 8) for n in TEAMS)
    assert not any(room(0, G, n) for G, n in ((4, 1), (4, 9), (0, 4), (9, 4)))


@pytest.mark.gpu
@pytest.mark.parametrize("B,n_kv,G,S", [(1, 2, 4, 40), (1, 1, 8, 129), (2, 2, 4, 384), (1, 1, 5, 768), (1, 1, 1, 3072), (1, 1, 4, 3100), (3, 1, 6, 1000), (10, 2, 4, 300)])
def test_pages(B, n_kv, G, S):
    import torch
    from gaac_b200 import Codec, attention
    from gaac_b200.kernel import workspace_error
    k16, v16 = O.kv_like(B * n_kv, S, 1), O.kv_like(B * n_kv, S, 2)
    k, v = to_bf16_cuda(k16), to_bf16_cuda(v16)
    kp, vp = Codec(n_kv).calibrate(k[:n_kv]).encode(k, "k"), Codec(n_kv).calibrate(v[:n_kv]).encode(v, "v")
    q16 = O.f32_to_bf16((np.random.default_rng(G).standard_normal((B, n_kv * G, 128)) * 0.1).astype(np.float32))
    o32 = torch.empty(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
    for nsplit in (1, 2, 3, 4, 5, 6, 7, 8, 9, 8, None):
        o32.fill_(float("nan"))
        out = attention(to_bf16_cuda(q16), kp, vp, SCALE, nsplit=nsplit, out_f32=o32)
        for b in range(B):
            ks, vs = (np.ascontiguousarray(x[b * n_kv:(b + 1) * n_kv].transpose(1, 0, 2)) for x in (k16, v16))
            assert_attention_close(o32[b].cpu().numpy(), q16[b], ks, vs, SCALE, (b, nsplit))
        assert torch.equal(out, o32.to(torch.bfloat16))
    assert not workspace_error("cuda")


@pytest.mark.gpu
def test_slots_longer_than_their_bound():
    """max_len only steers: rows of one launch that are longer than a team's ranges may be, beside others that are not, a padding row, rows that are all tail."""
    import torch
    import gaac_b200.kv_cache as kvc
    lens, n_kv, G = [3200, 300, 0, 7, 1537, 120], 1, 4
    cache, hist = kvc.CompressedKVCache(n_slots=len(lens), n_kv=n_kv, capacity=3216, bases=None), []
    for s, L in enumerate(lens):
        k, v = (np.ascontiguousarray(O.kv_like(n_kv, max(L, 1), 7 * s + i).transpose(1, 0, 2))[:L] for i in (1, 2))
        cache.prefill(s, to_bf16_cuda(k), to_bf16_cuda(v), check=False)
        hist.append((k, v))
    order = [0, 4, -1, 2, 1, 3, 5]
    q16 = O.f32_to_bf16((np.random.default_rng(3).standard_normal((len(order), n_kv * G, 128)) * 0.1).astype(np.float32))
    o32 = torch.empty(len(order), n_kv * G, 128, dtype=torch.float32, device="cuda")
    for nsplit in (2, 4, 8, 8, None):
        o32.fill_(float("nan"))
        cache.attention(to_bf16_cuda(q16), torch.tensor(order, dtype=torch.int32, device="cuda"), SCALE, max_len=300, nsplit=nsplit, out_f32=o32)
        for b, s in enumerate(order):
            if s < 0 or lens[s] == 0: assert not o32[b].any()
            else: assert_attention_close(o32[b].cpu().numpy(), q16[b], *hist[s], SCALE, (s, nsplit))
