"""Calls that fail although their kernels were queued (an error that an earlier call of the program left behind is reported by the launch that finds it): what they share with later calls, and
what the caller may free, is in order when they return."""
import ctypes
import numpy as np
import pytest
from common import to_bf16_cuda
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


def _leave_an_error_behind():
    """A CUDA call that is refused on the host and whose error nobody has taken."""
    assert _cudart().cudaSetDevice(9999) != 0


def _cudart():
    return ctypes.CDLL("libcudart.so.12")


def test_prompt_counters():
    import torch
    from gaac_b200 import CompressedKVCache, _lib
    n_kv, L, lib = 2, 300, _lib.lib()
    rows = [np.ascontiguousarray(O.kv_like(n_kv, L, seed=s).transpose(1, 0, 2)) for s in (1, 2)]
    rows[0] = np.full_like(rows[0], 0x3F80)          # its counts would outweigh those of any other prompt
    x, c = [to_bf16_cuda(r) for r in rows], CompressedKVCache(2, n_kv, L)
    ws = torch.zeros(lib.gaac_cache_tables_workspace_bytes(n_kv), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(lib.gaac_cache_prefill_scratch_bytes(L, n_kv), dtype=torch.uint8, device="cuda")
    stream = _lib.stream_ptr(torch.device("cuda", 0))
    call = lambda slot: lib.gaac_cache_prefill_own(c.k.c_store(), c.v.c_store(), x[slot].data_ptr(), x[slot].data_ptr(), L, n_kv * 128, slot, n_kv, c.tail_len.data_ptr(), c.S.data_ptr(),
                                                   c.cap, c.k.ovf_cap, 2 * n_kv, scratch.data_ptr(), scratch.numel(), c._slot_status.data_ptr() + 16 * slot, ws.data_ptr(), ws.numel(), stream)
    torch.cuda.synchronize()
    _leave_an_error_behind()
    assert call(0) != 0
    assert call(1) == 0
    for st in (c.k, c.v):
        b3, b4 = O.calibrate(np.ascontiguousarray(rows[1].transpose(1, 0, 2)), n_kv)
        assert np.array_equal(st.base3[n_kv:].cpu().numpy(), b3) and np.array_equal(st.base4[n_kv:].cpu().numpy(), b4)
    assert not bool(ws.any())


def test_encode_has_written_its_total():
    """A caller frees the total with a call that failed: by then the kernel that writes it has ended, although it was queued behind others."""
    import torch
    from gaac_b200 import Codec, _lib
    S, lib = 65536, _lib.lib()
    x16 = O.kv_like(1, S, seed=2)
    x = to_bf16_cuda(x16)
    c = Codec(1).calibrate(x)
    u8, i32 = dict(dtype=torch.uint8, device="cuda"), dict(dtype=torch.int32, device="cuda")
    sm, codes, slots = torch.empty(S * 128, **u8), torch.empty(S * 48, **u8), torch.empty(S // 16 * 1280, **u8)
    flags, sizes, off, ends = torch.empty(S, **i32), torch.empty(S // 16, **i32), torch.empty(S // 16, **i32), torch.empty(3, **i32)
    counter, total, work = torch.zeros(1, dtype=torch.int64, device="cuda"), torch.full((1,), 7, dtype=torch.int32, pin_memory=True), torch.zeros(1 << 28, **u8)
    call = lambda: lib.gaac_encode_queued(x.data_ptr(), 1, S, S, S, c.base3.data_ptr(), c.base4.data_ptr(), None, 1, 0, sm.data_ptr(), codes.data_ptr(), flags.data_ptr(), slots.data_ptr(),
                                          sizes.data_ptr(), off.data_ptr(), ends.data_ptr() + 8, ends.data_ptr(), total.data_ptr(), counter.data_ptr(), stream)
    stream = _lib.stream_ptr(torch.device("cuda", 0))
    torch.cuda.synchronize()
    for _ in range(10): work.add_(1)                 # about a millisecond
    _leave_an_error_behind()
    assert call() != 0
    n = int(total)
    page = c.encode(x, "k")
    assert n == int(page.ovf_head_start[-1]) and int(counter) == 0
    assert call() == 0 and lib.gaac_wait_total(total.data_ptr(), stream) == 0 and int(total) == n


def test_encode_is_refused_in_a_capture_of_a_stream_that_has_encoded():
    """.. before anything of it is captured: the graph goes on without it."""
    import torch
    from gaac_b200 import Codec
    x = to_bf16_cuda(O.kv_like(2, 100, seed=2))
    c, side, graph, y = Codec(2).calibrate(x), torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros(4, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        c.encode(x, "k")
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        with pytest.raises(RuntimeError, match="cannot be captured"):
            c.encode(x, "k")
        assert c.encode(x[:0], "k").S == 100         # (no heads: no kernels)
        y.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert y.tolist() == [1.0] * 4


def test_encode_is_refused_in_a_capture_whatever_the_allocators_hold():
    """A first encode on the stream, and one whose total finds no page-locked word free: the graph goes on without either."""
    import torch
    from gaac_b200 import Codec
    x = to_bf16_cuda(O.kv_like(2, 100, seed=2))
    for first in (True, False):
        c, side, graph, y = Codec(2).calibrate(x), torch.cuda.Stream(priority=-1), torch.cuda.CUDAGraph(), torch.zeros(4, device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            if not first: c.encode(x, "k")
            ref = c.encode(x, "v") if not first else None
        words = [torch.empty(1, dtype=torch.int32, pin_memory=True) for _ in range(200)]
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            with pytest.raises(RuntimeError, match="cannot be captured"):
                c.encode(x, "k")
            y.add_(1)
        graph.replay()
        torch.cuda.synchronize()
        assert y.tolist() == [1.0] * 4 and len(words) == 200
        with torch.cuda.stream(side):
            page = c.encode(x, "v")
        torch.cuda.synchronize()
        assert ref is None or torch.equal(page.ovf, ref.ovf)


def test_wait_for_a_total_takes_its_error():
    """A stream that is being captured cannot be asked: the wait says so, and no later launch does."""
    import torch
    from gaac_b200 import _lib
    side, word, graph, rt = torch.cuda.Stream(), ctypes.c_int32(-1), ctypes.c_void_p(), _cudart()
    stream = ctypes.c_void_p(side.cuda_stream)
    assert rt.cudaStreamBeginCapture(stream, 2) == 0
    try:
        assert _lib.lib().gaac_wait_total(ctypes.byref(word), stream) == 4
        assert rt.cudaPeekAtLastError() == 0
    finally:
        assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) != 0        # the question ended the capture
        rt.cudaGetLastError()
