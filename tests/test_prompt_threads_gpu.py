"""Prompt tables while two host threads prefill caches of their own on one stream, with one set of the counters that a call leaves zero (as CompressedKVCache shares them): the launches
of two calls must not come in between each other."""
import threading
import numpy as np
import pytest
from common import to_bf16_cuda
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_kv,L,slots", [(2, 300, 500), (1, 40000, 50)])        # 2 x 40000: more than a 16-bit count holds
def test_two_threads_on_one_stream(n_kv, L, slots):
    import torch
    from gaac_b200 import CompressedKVCache, _lib
    rows = [np.ascontiguousarray(O.kv_like(n_kv, L, seed=s).transpose(1, 0, 2)) for s in (1, 2)]
    rows[1] = ((rows[1] & 0x807F) | ((((rows[1] >> 7) & 0xFF) // 2 + 20) << 7)).astype(np.uint16)         # exponents of a range of their own
    dev, caches, lib = [to_bf16_cuda(r) for r in rows], [CompressedKVCache(slots, n_kv, L) for _ in rows], _lib.lib()
    ws = torch.zeros(lib.gaac_cache_tables_workspace_bytes(n_kv), dtype=torch.uint8, device="cuda")
    scratch = [torch.empty(lib.gaac_cache_prefill_scratch_bytes(L, n_kv), dtype=torch.uint8, device="cuda") for _ in rows]
    codes, together = [set(), set()], threading.Barrier(2)
    torch.cuda.synchronize()

    def work(i):                                     # every pass fills a slot of its own, so every pass's tables are there at the end
        c, x, status = caches[i], dev[i].data_ptr(), caches[i]._slot_status.data_ptr()
        K, V, stream = c.k.c_store(), c.v.c_store(), _lib.stream_ptr(torch.device("cuda", 0))
        args = (c.tail_len.data_ptr(), c.S.data_ptr(), c.cap, c.k.ovf_cap, c.k.base3.shape[0], scratch[i].data_ptr(), scratch[i].numel())
        kept = ws.data_ptr(), ws.numel(), stream
        together.wait()
        for slot in range(slots):
            codes[i].add(lib.gaac_cache_prefill_own(K, V, x, x, L, n_kv * 128, slot, n_kv, *args, status + 16 * slot, *kept))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads: t.start()
    for t in threads: t.join()
    assert codes == [{0}, {0}]
    for c, r, x in zip(caches, rows, dev):
        want = O.calibrate(np.ascontiguousarray(r.transpose(1, 0, 2)), n_kv)
        for st in (c.k, c.v):
            for got, ref in zip((st.base3, st.base4), want):
                assert np.array_equal(got.cpu().numpy(), np.tile(ref, (slots, 1)))
        assert all(torch.equal(t.view(torch.int16), x.view(torch.int16)) for t in c.decompress(slots - 1))
    assert not bool(ws.any())
