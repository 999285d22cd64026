"""The attention workspace of a stream: a captured CUDA graph keeps the address it was captured with, so a workspace that a later call outgrows stays alive."""
import gc
import weakref
import numpy as np
import pytest
from common import to_bf16_cuda, assert_attention_close
from oracle import gaac_oracle as O


def test_outgrown_workspaces_stay_and_are_bounded(monkeypatch):
    import types
    import torch
    import gaac_b200.kernel as K
    monkeypatch.setattr(K, "_WS", {})
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: types.SimpleNamespace(cuda_stream=7))
    shapes = [(64, 8, 2), (32, 8, 117), (8, 64, 18), (32, 64, 40), (1, 32, 200), (64, 64, 33), (2, 9000, 1), (4, 9000, 1), (2, 9000, 3), (64, 8, 2)]
    seen, biggest = [], {}
    for B, n_q, ns in shapes:
        ws = K.workspace("cpu", B, n_q, ns)
        need = K._lib.lib().gaac_attn_workspace_bytes(B, n_q, ns)
        assert ws.numel() >= need and not ws.any()
        seen.append(weakref.ref(ws))
        big = B * n_q if B * n_q > 16320 else 0
        biggest[big] = max(biggest.get(big, 1 << 20), ws.numel())
    del ws
    gc.collect()
    assert all(r() is not None for r in seen)
    for big, most in biggest.items():
        assert sum(t.numel() for t in K._WS[(None, 7, big)]) < 2 * most
    assert K.workspace("cpu", 64, 8, 2) is seen[5]() and K.workspace("cpu", 2, 9000, 2) is seen[8]() is not seen[7]()       # shapes above the fixed header share nothing


def test_stream_pointer_takes_every_form_of_a_device(monkeypatch):
    import types
    import torch
    from gaac_b200 import _lib
    asked = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: (asked.append(dev), types.SimpleNamespace(cuda_stream=7))[1])
    monkeypatch.setattr(_lib, "_raw_stream", lambda index: 100 + index)
    assert _lib.stream_ptr(torch.device("cuda", 1)) == 101 and not asked
    forms = [None, "cuda", "cuda:0", 0, torch.device("cuda"), torch.device("cpu")]
    assert [_lib.stream_ptr(d) for d in forms] == [7] * len(forms) and asked == forms


@pytest.mark.gpu
def test_graphs_of_descending_batch_sizes():
    """Graphs captured for 64 rows, then 32, then 4 on one stream; then what the allocator would have got back is overwritten, and all are replayed."""
    import torch
    from gaac_b200 import CompressedKVCache
    n_kv, G, L = 1, 8, 900
    k16, v16 = (np.ascontiguousarray(O.kv_like(n_kv, L, i).transpose(1, 0, 2)) for i in (1, 2))
    cache = CompressedKVCache(n_slots=64, n_kv=n_kv, capacity=32768, bases=None)
    for s in range(64):
        cache.prefill(s, to_bf16_cuda(k16), to_bf16_cuda(v16), check=False)
    cache.settle_prefills()
    q16 = O.f32_to_bf16((np.random.default_rng(0).standard_normal((64, n_kv * G, 128)) * 0.1).astype(np.float32))
    q = to_bf16_cuda(q16)
    stream, graphs = torch.cuda.Stream(), []
    with torch.cuda.stream(stream):
        for B in (64, 32, 4):
            o32 = torch.zeros(B, n_kv * G, 128, dtype=torch.float32, device="cuda")
            slots = torch.arange(B, dtype=torch.int32, device="cuda")
            call = lambda: cache.attention(q[:B], slots, 128 ** -0.5, max_len=32768, out_f32=o32)
            call()
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                call()
            graphs.append((B, g, o32))
        junk = [torch.full((n,), 0x5A, dtype=torch.uint8, device="cuda") for n in (1 << 20, 1 << 21, 5 << 20, 16 << 20, 20 << 20) for _ in range(3)]
        for B, g, o32 in graphs + graphs[::-1]:
            o32.zero_()
            g.replay()
            torch.cuda.synchronize()
            for b in (0, B - 1):
                assert_attention_close(o32[b].cpu().numpy(), q16[b], k16, v16, 128 ** -0.5, (B, b))
        assert all(bool((t == 0x5A).all()) for t in junk)          # and no replay wrote into anybody else's memory


@pytest.mark.gpu
@pytest.mark.parametrize("B,n_kv,L", [(1, 8, 40), (3, 8, 200), (40, 4, 70)])
def test_no_wait_runs_out_in_short_launches(B, n_kv, L):
    """Launches whose first stages are published a few cycles after the ring was cleared (grid, ranges by length, one wave): a word that was cleared late would leave its
    tiles out and set the error word."""
    import torch
    from gaac_b200 import CompressedKVCache
    from gaac_b200.kernel import workspace_error
    k16, v16 = (np.ascontiguousarray(O.kv_like(n_kv, L, i).transpose(1, 0, 2)) for i in (1, 2))
    cache = CompressedKVCache(n_slots=B, n_kv=n_kv, capacity=4096, bases=None)
    for s in range(B):
        cache.prefill(s, to_bf16_cuda(k16), to_bf16_cuda(v16), check=False)
    q16 = O.f32_to_bf16((np.random.default_rng(0).standard_normal((B, 4 * n_kv, 128)) * 0.1).astype(np.float32))
    q, slots = to_bf16_cuda(q16), torch.arange(B, dtype=torch.int32, device="cuda")
    refs = {}
    for b in {0, B - 1}:                                                        # every call is held against the oracle, on the device
        ref, mag = O.attention_ref(q16[b], k16, v16, 128 ** -0.5, with_abs=True)
        refs[b] = torch.from_numpy(ref).cuda(), torch.from_numpy(O.attention_bound(mag)).cuda()
    worst = torch.zeros((), dtype=torch.float64, device="cuda")
    for i in range(300):
        o32 = torch.empty(B, 4 * n_kv, 128, dtype=torch.float32, device="cuda")
        cache.attention(q, slots, 128 ** -0.5, max_len=(L, 4096, None)[i % 3], nsplit=None if i % 4 else 1, out_f32=o32)
        for b, (ref, bound) in refs.items():
            worst = torch.maximum(worst, ((o32[b].double() - ref).abs() / bound).max())
    assert not workspace_error("cuda:0") and float(worst) <= 1.0
