"""Escape streams longer than 31 bits count: offsets that have run over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
