"""Argument checks of the entry points that keep counters between calls: refused before any launch."""
import ctypes
import pytest


@pytest.fixture(scope="module")
def lib():
    from gaac_b200 import build, _lib
    build.build()
    return _lib.lib()


def test_encode_queued_and_wait(lib):
    z, fake, word = ctypes.c_void_p(0), ctypes.c_void_p(0x1000), ctypes.c_int32(7)
    w = ctypes.cast(ctypes.byref(word), ctypes.c_void_p)
    args = lambda total, counter, x=fake: (x, 1, 16, 16, 16, fake, fake, z, 1, 0, fake, fake, fake, fake, fake, fake, fake, fake, total, counter, z)
    assert lib.gaac_encode_queued(*args(z, fake)) == 1 and lib.gaac_encode_queued(*args(w, z)) == 1
    assert lib.gaac_encode_queued(*args(w, ctypes.c_void_p(0x1004))) == 3
    assert word.value == 7                                                      # a call that is refused does not touch the word ..
    assert lib.gaac_encode_queued(*args(w, fake, z)) == 1
    assert lib.gaac_wait_total(z, z) == 1
    word.value = 5
    assert lib.gaac_wait_total(w, z) == 0                                       # .. and one that is there needs no GPU


def test_prefill_own(lib):
    from gaac_b200 import _lib
    f, z = ctypes.c_void_p(0x1000), ctypes.c_void_p(0)
    st = _lib.Store(*[0x1000] * 9)
    need, ws = lib.gaac_cache_prefill_scratch_bytes(100, 2), lib.gaac_cache_tables_workspace_bytes(2)
    assert ws == 2 * 2 * 128 * 512 and lib.gaac_cache_tables_workspace_bytes(0) == 0
    assert need >= 2 * 2 * 6 * 1284

    def call(L=100, rows=4, scratch=need, work=ws, at=f, slot=1, k=f):
        return lib.gaac_cache_prefill_own(st, st, k, f, L, 256, slot, 2, f, f, 112, 4096, rows, f, scratch, f, at, work, z)
    assert call(L=0) == 1 and call(L=113) == 1 and call(rows=3) == 1 and call(slot=-1) == 1 and call(k=z) == 1 and call(at=z) == 1 and call(scratch=need - 1) == 1
    assert call(work=ws - 1) == 5 and call(at=ctypes.c_void_p(0x1008)) == 3
