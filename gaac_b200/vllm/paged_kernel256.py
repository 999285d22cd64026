"""Decode attention over the paged block buffer, head_dim 256 (mirror of gaac/vllm/paged_kernel256.py).

A 256-dim head is stored as two 128-dim half-heads in neighbouring tile slots of a block, each half-head with its own exponent
bases: the store (LayerState with n_kv = 2 * kv heads), the block decoder and the bases all work on half-heads, only this
kernel puts the halves together.  In the kernel two warps share one stream of tiles, one per half: each rebuilds its half of the K
tile, the two partial scores meet in shared memory, both warps run the same softmax step and each accumulates the 128 output
dimensions of its half of V.
"""
from __future__ import annotations
import torch
from .. import _lib
from ..kernel import SM_COUNT_B200, workspace, choose_flat256, choose_nsplit256, _flat_splits


def paged_attention256(q, out, buf, raw, mt, bt, seq_lens, bases, TS, n_q, n_kv, nsplit=None, scale=None, out_f32=None):
    """q: [B, n_q, 256] bf16 contiguous; out: [B, n_q*256] bf16 (written); n_kv: 256-dim kv heads; bases: (b3k, b4k, b3v, b4v) uint8
    [2*n_kv, 128], one row per half-head; the other arguments as paged_attention.  scale defaults to 1/sqrt(256).
    (gaac/vllm/paged_kernel256.py:299-305)"""
    B = q.shape[0]
    G = n_q // max(1, n_kv)
    if q.shape[-1] != 256: raise RuntimeError("head_dim must be 256")
    if not (1 <= G <= 8 and G * n_kv == n_q): raise RuntimeError("GQA group size must be 1..8")
    if TS % 16: raise RuntimeError("tile stride must be a multiple of 16")
    if not q.is_cuda: raise RuntimeError("gaac_b200 attention needs CUDA tensors: there is no CPU path")
    bt_stride = _lib.row_stride(bt)
    flat = 0
    if nsplit is None:
        nsplit = choose_nsplit256(B, n_kv, bt.shape[1] * 16, group=G)
        flat = choose_flat256(B, n_kv, bt.shape[1] * 16, bt_stride * 16, SM_COUNT_B200, G)
        if flat: nsplit = _flat_splits(B, n_kv, flat)                                          # what the workspace must have room for
    st = (buf, raw, mt, None, None, None, bases[0], bases[1], bases[2], bases[3], 2 * n_kv, TS, TS - 2880)
    stream = _lib.stream_ptr(q.device)
    ws = workspace(q.device, B, 2 * n_q, nsplit, stream)
    name = "gaac_paged_decode_attn256_flat" if flat else "gaac_paged_decode_attn256"
    _lib.check(getattr(_lib.host(), name)(st, bt, bt_stride, seq_lens, q, B, n_q, float(scale) if scale is not None else 256 ** -0.5, flat or int(nsplit), ws, ws.numel(), out, out_f32, stream), name)
    return out
