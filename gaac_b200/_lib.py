"""ctypes binding of libgaac_b200.so (the C ABI declared in include/gaac_b200.h).

There is no fallback: if the library is missing or a call fails, a RuntimeError is raised.
"""
from __future__ import annotations
import ctypes as C
import os
import threading
import weakref

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.environ.get("GAAC_B200_LIB") or os.path.join(_HERE, "libgaac_b200.so")     # GAAC_B200_LIB: use a library built elsewhere
_lib = None

vp, i32, i64, f32, sz = C.c_void_p, C.c_int, C.c_int64, C.c_float, C.c_size_t


class Side(C.Structure):
    """gaac_side"""
    _fields_ = [("sm", vp), ("codes", vp), ("flags", vp), ("tile_off", vp), ("ovf", vp), ("head_start", vp),
                ("ovf_bytes", i64), ("base3", vp), ("base4", vp), ("tail", vp)]


class Store(C.Structure):
    """gaac_store"""
    _fields_ = [("sm", vp), ("codes", vp), ("flags", vp), ("tile_off", vp), ("ovf", vp), ("ovf_used", vp), ("tail", vp),
                ("base3", vp), ("base4", vp)]


class Paged(C.Structure):
    """gaac_paged"""
    _fields_ = [("buf", vp), ("raw", vp), ("mt", vp), ("stack", vp), ("top", vp), ("err", vp),
                ("b3k", vp), ("b4k", vp), ("b3v", vp), ("b4v", vp), ("n_kv", i32), ("TS", i32), ("ovf_slot", i32)]


class Exchange(C.Structure):
    """gaac_exchange"""
    _fields_ = [("recv", vp), ("epoch", vp), ("ticket", vp), ("err", vp), ("rank", i32), ("world", i32), ("rows_cap", i32)]


_SIGNATURES = {
    "gaac_status_string": (C.c_char_p, [i32]),
    "gaac_abi_version": (i32, []),
    "gaac_encode_tiles": (i32, [vp, i64, i64, i64, i64, vp, vp, vp, i32, i32, vp, vp, vp, vp, vp, vp]),
    "gaac_compact": (i32, [vp, vp, i64, i64, vp, vp, vp, i64, vp, vp, i64, i64, vp, vp]),
    "gaac_head_prefix": (i32, [vp, i64, vp, vp]),
    "gaac_encode_begin": (i32, [vp, i64, i64, i64, i64, vp, vp, vp, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, vp]),
    "gaac_encode_sized": (i32, [vp, i64, i64, i64, i64, vp, vp, vp, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp]),
    "gaac_encode_queued": (i32, [vp, i64, i64, i64, i64, vp, vp, vp, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp]),
    "gaac_wait_total": (i32, [vp, vp]),
    "gaac_compact_copy": (i32, [vp, vp, i64, i64, vp, vp, vp, i64, vp, i64, i64, vp, i32, i64, i64, vp, vp]),
    "gaac_decode_page": (i32, [vp, vp, vp, vp, i64, vp, vp, vp, vp, vp, i32, i32, i64, i64, i64, vp, vp]),
    "gaac_exponent_hist": (i32, [vp, i64, i64, vp, vp]),
    "gaac_bases_from_hist": (i32, [vp, i64, vp, vp, vp]),
    "gaac_set_launch_overlap": (None, [i32]),
    "gaac_attn_workspace_bytes": (sz, [i32, i32, i32]),
    "gaac_attn_workspace_header_bytes": (sz, [i32, i32]),
    "gaac_decode_attn_pages": (i32, [C.POINTER(Side), C.POINTER(Side), vp, i32, i32, i32, i64, i64, f32, i32, i32, vp, sz, vp, vp, vp, C.POINTER(Exchange), i32, vp]),
    "gaac_decode_attn_exchange": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, sz, C.POINTER(Exchange), vp, vp, vp]),
    "gaac_debug_decode_attn_rebuild": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, i64, f32, i32, vp, i32, i32, vp, sz, vp, vp, vp, vp, i64, vp]),
    "gaac_debug_paged_decode_attn_rebuild": (i32, [C.POINTER(Paged), vp, i64, vp, vp, i32, i32, f32, i32, vp, sz, vp, vp, vp, vp, i64, vp]),
    "gaac_debug_team_room": (i32, [i32, i32, i32]),
    "gaac_decode_attn": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, sz, vp, vp, vp]),
    "gaac_decode_attn_partial": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, sz, vp, vp]),
    "gaac_combine": (i32, [vp, vp, vp, i64, i32, vp, vp, vp]),
    "gaac_combine_parts": (i32, [vp, i64, i32, vp, vp, vp]),
    "gaac_decode_attn_push": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, sz, C.POINTER(Exchange), vp]),
    "gaac_exchange_merge": (i32, [C.POINTER(Exchange), i64, vp, vp, vp]),
    "gaac_append_kv": (i32, [C.POINTER(Store), C.POINTER(Store), vp, vp, vp, i32, i32, vp, vp, i64, i64, i32, vp, vp]),
    "gaac_cache_calibrate_scratch_bytes": (C.c_size_t, [i32]),
    "gaac_cache_calibrate": (i32, [C.POINTER(Store), C.POINTER(Store), vp, vp, i64, i64, i32, i32, i32, vp, C.c_size_t, vp]),
    "gaac_cache_prefill_scratch_bytes": (C.c_size_t, [i64, i32]),
    "gaac_cache_prefill": (i32, [C.POINTER(Store), C.POINTER(Store), vp, vp, i64, i64, i32, i32, vp, vp, i64, i64, i32, vp, C.c_size_t, vp, i32, vp]),
    "gaac_cache_tables_workspace_bytes": (C.c_size_t, [i32]),
    "gaac_cache_prefill_own": (i32, [C.POINTER(Store), C.POINTER(Store), vp, vp, i64, i64, i32, i32, vp, vp, i64, i64, i32, vp, C.c_size_t, vp, vp, C.c_size_t, vp]),
    "gaac_paged_store": (i32, [C.POINTER(Paged), vp, vp, i64, i64, vp, i32, vp, vp]),
    "gaac_paged_release": (i32, [C.POINTER(Paged), vp, i32, vp]),
    "gaac_paged_decode_blocks": (i32, [C.POINTER(Paged), vp, i32, vp, vp, i64, vp]),
    "gaac_paged_decode_attn": (i32, [C.POINTER(Paged), vp, i64, vp, vp, i32, i32, f32, i32, vp, sz, vp, vp, vp]),
    "gaac_paged_decode_attn256": (i32, [C.POINTER(Paged), vp, i64, vp, vp, i32, i32, f32, i32, vp, sz, vp, vp, vp]),
    "gaac_decode_attn_balanced": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, sz, vp, vp, vp]),
    "gaac_paged_decode_attn_balanced": (i32, [C.POINTER(Paged), vp, i64, vp, vp, i32, i32, f32, i32, vp, sz, vp, vp, vp]),
    "gaac_decode_attn_flat": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, sz, vp, vp, vp]),
    "gaac_paged_decode_attn_flat": (i32, [C.POINTER(Paged), vp, i64, vp, vp, i32, i32, f32, i32, vp, sz, vp, vp, vp]),
    "gaac_paged_decode_attn256_flat": (i32, [C.POINTER(Paged), vp, i64, vp, vp, i32, i32, f32, i32, vp, sz, vp, vp, vp]),
    "gaac_decode_attn_static": (i32, [C.POINTER(Side), C.POINTER(Side), vp, vp, i32, i32, i32, vp, i64, f32, i32, vp, i32, i32, vp, vp, vp]),
    "gaac_static_workspace_bytes": (sz, []),
    "gaac_static_workspace_error": (i32, [vp, i32, vp]),
}
EXPORTS = tuple(_SIGNATURES)
ABI_VERSION = 4


def lib():
    """The loaded library.  Raises RuntimeError when it has not been built (python -m gaac_b200.build)."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(f"{LIB_PATH} is missing: build it with `python -m gaac_b200.build` (needs nvcc); there is no fallback path")
        L = C.CDLL(LIB_PATH)
        for name, (res, args) in _SIGNATURES.items():
            fn = getattr(L, name)
            fn.restype, fn.argtypes = res, args
        if L.gaac_abi_version() != ABI_VERSION:
            raise RuntimeError(f"{LIB_PATH} has ABI version {L.gaac_abi_version()}, this package binds version {ABI_VERSION}: rebuild it (python -m gaac_b200.build --force)")
        _lib = L
    return _lib


_load, _host = lib, None


def host():
    """The module whose functions are the library's hot ones and take tensors as they are (csrc/gaac_host.cpp).  Like the library it has no substitute."""
    global _host
    if _host is None:
        import torch                                 # (its libraries are what the module is linked to)
        handle = _load()._handle
        try:
            from . import _host as module
        except ImportError as e:
            raise RuntimeError(f"gaac_b200's module _host is missing or does not fit this torch ({torch.__version__}): build it with `python -m gaac_b200.build`") from e
        wanted = f"ABI {ABI_VERSION}, torch {torch.__version__}"                       # (it passes arguments as the header and torch's classes were when it was made)
        found = getattr(module, "built_for", "nobody knows what")                      # (one from before it said so, under the name without an interpreter)
        if found != wanted:
            raise RuntimeError(f"{module.__file__} was built for {found}, not for {wanted}: rebuild it with `python -m gaac_b200.build`")
        module.bind(handle)
        _host = module
    return _host


def check(status: int, what: str):
    if status != 0:
        raise RuntimeError(f"{what}: {lib().gaac_status_string(status).decode()} (status {status})")


def row_stride(t) -> int:
    """Stride of dim 0 in elements as the library wants it.  torch is free to report anything for a dimension of size 1 (a
    one-row tensor often comes back with the stride of its second dimension), and the library checks the stride against the row
    width: a tensor with at most one row gets the width of a packed row instead."""
    if t.shape[0] > 1:
        return t.stride(0)
    n = 1
    for s in t.shape[1:]:
        n *= s
    return max(n, 1)


class _Buffers(dict):                                # (device index, stream) -> buffer, oldest first
    __slots__ = ("__weakref__",)

    def __reduce__(self):                            # copied and pickled with its user as None: the copy asks for itself
        return type(None), ()


class Kept:
    """Zeroed device buffers that every call leaves zero, so that one per stream serves all objects that make such calls.  They live as long as one of the objects that have
    asked for them (which hold them as `_kept`, or None until then); beyond MOST streams the oldest goes.  A buffer that goes is the allocator's again on the stream that it was made and used on; the
    caller holds what it was given until its launches are queued, since another thread's call may drop it here."""
    MOST = 32

    def __init__(self, dtype: str):
        self._dtype, self._now, self._lock = dtype, lambda: None, threading.RLock()

    def join(self) -> _Buffers:
        """What a user holds as `_kept`."""
        with self._lock:
            buffers = self._now()
            if buffers is None:
                buffers = _Buffers()
                self._now = weakref.ref(buffers)
        return buffers

    def of(self, user, dev, stream: int, n: int):
        """n or more elements for `user`'s calls on the current stream of dev, which must not be capturing (they would be zero only when the graph runs)."""
        buffers = user._kept
        if buffers is None:
            buffers = user._kept = self.join()
        t = buffers.get((dev.index, stream))
        if t is None or t.numel() < n:
            import torch
            t = torch.zeros(n, dtype=getattr(torch, self._dtype), device=dev)
            with self._lock:
                buffers.pop((dev.index, stream), None)
                buffers[dev.index, stream] = t
                while len(buffers) > self.MOST:
                    del buffers[next(iter(buffers))]
        return t

    def values(self) -> list:
        return list((self._now() or {}).values())

    def __len__(self):
        return len(self._now() or ())


ENCODE_COUNTERS = Kept("int64")       # the word that the encoder's CTAs count themselves in
TABLE_COUNTERS = Kept("uint8")        # counters of a prompt's tables, 128 KB per kv head


def capturing() -> bool:
    """torch.cuda.is_current_stream_capturing without the Python function around it."""
    global capturing
    import torch
    capturing = getattr(torch._C, "_cuda_isCurrentStreamCapturing", torch.cuda.is_current_stream_capturing)
    return capturing()


def ptr(t):
    """Device pointer of a tensor (None -> NULL)."""
    return None if t is None else t.data_ptr()


def stream_ptr(device=None):
    """The current stream of a device.  torch.cuda.current_stream makes a Stream object, 2.3 us of the ten or so that a call of this package costs; the function
    underneath it takes 0.1 us."""
    index = getattr(device, "index", None)
    if type(index) is int and device.type == "cuda":           # (a string's `index` is a method; "cuda:0", a number or None take the way below)
        return _raw_stream(index)
    import torch
    return torch.cuda.current_stream(device).cuda_stream


def _raw_stream(index):
    global _raw_stream
    import torch
    _raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda i: torch.cuda.current_stream(i).cuda_stream)
    return _raw_stream(index)
