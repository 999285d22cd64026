"""Escape streams longer than 31 bits count: the encoder's counters, which such sums are put into as if earlier CTAs had them, and offsets that have run over."""
import numpy as np
import pytest
from common import to_bf16_cuda
from oracle import gaac_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1, 1 << 31, (1 << 31) + 77, 1 << 33])       # bytes beyond the 2^31 - 1 that a total can be
def test_totals(more):
    import torch
    from gaac_b200 import Codec, _lib
    S, H, lib, stream = 21 * 16, 3, _lib.lib(), _lib.stream_ptr(torch.device("cuda", 0))        # six CTAs per head
    x16 = O.kv_like(H, S, seed=2)
    x = to_bf16_cuda(x16)
    c = Codec(H).calibrate(x)
    n = int(c.encode(x, "k").ovf_head_start[-1])
    u8, i32 = dict(dtype=torch.uint8, device="cuda"), dict(dtype=torch.int32, device="cuda")
    sm, codes, slots = torch.empty(H * S * 128, **u8), torch.empty(H * S * 48, **u8), torch.empty(H * S // 16 * 1280, **u8)
    flags, sizes, off, sums, ends = torch.empty(H * S, **i32), torch.empty(H * S // 16, **i32), torch.empty(H * S // 16, **i32), torch.empty(H, **i32), torch.empty(H + 1, **i32)
    counter, total = torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, pin_memory=True)

    def call():
        assert lib.gaac_encode_queued(x.data_ptr(), H, S, S, S, c.base3.data_ptr(), c.base4.data_ptr(), None, H, 0, sm.data_ptr(), codes.data_ptr(), flags.data_ptr(), slots.data_ptr(),
                                      sizes.data_ptr(), off.data_ptr(), sums.data_ptr(), ends.data_ptr(), total.data_ptr(), counter.data_ptr(), stream) == 0
        return lib.gaac_wait_total(total.data_ptr(), stream), int(total)
    counter.fill_(2 ** 31 - 1 - n + more)
    assert call() == ((0, 2 ** 31 - 1) if more == 0 else (1, -2))
    torch.cuda.synchronize()
    assert int(counter) == 0 and call() == (0, n)


def test_offsets_below_zero_are_not_written():
    """Where head_start or tile_off have run over 31 bits, the tiles are refused, and the padding behind the last head."""
    import torch
    from gaac_b200 import _lib
    lib, stream = _lib.lib(), _lib.stream_ptr(torch.device("cuda", 0))
    H, ntiles, size, front = 3, 5, 40, 4096
    slots = torch.full((H * ntiles, 1280), 7, dtype=torch.uint8, device="cuda")
    sizes = torch.full((H, ntiles), size, dtype=torch.int32, device="cuda")
    off = torch.arange(ntiles, dtype=torch.int32, device="cuda").mul(size).repeat(H, 1)
    off[2, 3] = -1000
    start = torch.tensor([0, -2000, 200, -500], dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    buf = torch.full((front + 600,), 0x5A, dtype=torch.uint8, device="cuda")     # the stream begins behind `front` bytes, so that nothing can leave the buffer
    _lib.check(lib.gaac_compact_copy(slots.data_ptr(), sizes.data_ptr(), H, ntiles, start.data_ptr(), buf.data_ptr() + front, off.data_ptr(), ntiles, None, 0, 0, None, 8, 600, 0,
                                     status.data_ptr(), stream), "gaac_compact_copy")
    want = np.full(front + 600, 0x5A, np.uint8)
    for h, t in [(0, t) for t in range(ntiles)] + [(2, 0), (2, 1), (2, 2), (2, 4)]:
        at = front + (0, None, 200)[h] + size * t
        want[at:at + size] = 7
    assert np.array_equal(buf.cpu().numpy(), want) and int(status) == 1
