"""What this package does for its users, as cases that can be timed: decode steps over the three cache forms (a pair of Pages, the
slot cache, the paged block buffer), and the work around them (encode, decode, prompt prefill, chunked prefill).

A case is a dict of plain values with a `path`:

  pages     attention() over two Pages: B sequences of S tokens each
  slots     one decode step of CompressedKVCache: append of one token per row, attention; lengths differ from row to row
  paged     one decode step of the paged layout: LayerState.store of one token per sequence, paged_attention (or the head_dim 256 form)
  encode    Codec.encode of a K and a V tensor [n_kv, S, 128]
  decode    Codec.decode of the two Pages back to BF16
  prefill   CompressedKVCache.prefill of `B` prompts
  chunk     chunked prefill of the paged layout: the context so far is expanded with LayerState.decode_blocks, a chunk of new tokens stored

The values are the ones of gaac_b200.synth: Gaussian with a log-normal scale per channel, one in ten groups wide, one in five hundred raw.

A decode step changes its cache, so a pass starts by putting the counters back to where they stood before the step (one small
launch), as a program does that drops a drafted token: the same step can then be taken any number of times, the rows whose block
fills (one in sixteen) included.
"""
import math
import random

import numpy as np
import torch

from gaac_b200 import Codec, CompressedKVCache, attention
from gaac_b200.synth import synth_kv
from gaac_b200.vllm.paged_kernel import paged_attention
from gaac_b200.vllm.paged_kernel256 import paged_attention256
from gaac_b200.vllm.store import OVF_OFF, LayerState

D, T = 128, 16
OVF_SLOT = 128                  # escape bytes per tile slot of the paged layout
SCALE = D ** -0.5
# bytes per (token, kv head, kind) of the compressed form: sign/mantissa, codes, tag word, tile offset, and the escape bytes of these values
COMPRESSED = 128 + 48 + 4 + 0.25 + 3.3
PLAIN = 256


def listed():
    return [
        # batch 1 over two Pages, 32 query / 8 kv heads: the first tokens of a chat (latency), and the 64K context
        {"name": "pages_1x500", "path": "pages", "B": 1, "n_kv": 8, "group": 4, "S": 500},
        {"name": "pages_1x65536", "path": "pages", "B": 1, "n_kv": 8, "group": 4, "S": 65536},
        # slot cache: an interactive batch with a padding row, as a captured batch size has; and large-batch serving, 64 query / 8 kv
        # heads sharded to one kv head per GPU
        {"name": "slots_7x3000", "path": "slots", "B": 7, "pad": 1, "n_kv": 8, "group": 4, "lo": 200, "hi": 3000, "own": False},
        {"name": "slots_64x32768", "path": "slots", "B": 64, "pad": 0, "n_kv": 1, "group": 8, "lo": 32000, "hi": 32768, "own": True},
        # paged layout: a handful of short sequences, the 16 ragged sequences of the serving benchmark, head_dim 256
        {"name": "paged_5x1500", "path": "paged", "B": 5, "n_kv": 8, "group": 4, "lo": 40, "hi": 1500, "wide": False},
        {"name": "paged_16x65536", "path": "paged", "B": 16, "n_kv": 8, "group": 4, "lo": 4096, "hi": 65536, "wide": False},
        {"name": "paged256_8x8192", "path": "paged", "B": 8, "n_kv": 4, "group": 4, "lo": 1024, "hi": 8192, "wide": True},
        # encoder: a prompt of odd length, and the 64K context
        {"name": "encode_8x1111", "path": "encode", "n_kv": 8, "S": 1111},
        {"name": "encode_8x65536", "path": "encode", "n_kv": 8, "S": 65536},
        # the stored context back to BF16
        {"name": "decode_8x65536", "path": "decode", "n_kv": 8, "S": 65536},
        # three prompts of one scheduler step, each calibrated on itself
        {"name": "prefill_3x4001", "path": "prefill", "B": 3, "n_kv": 8, "L": 4001, "own": True},
        # the fourth chunk of 2048 tokens (the last one short) of a prompt
        {"name": "chunk_6144+1500", "path": "chunk", "n_kv": 8, "context": 6144, "new": 1500},
    ]


def _log_int(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(("pages", "pages", "slots", "slots", "paged", "paged", "encode", "decode", "prefill", "chunk"))
    n_kv, group = rng.choice((1, 2, 4, 8)), rng.choice((1, 4, 4, 5, 6, 8))
    most = 1 << 20                                          # (token, kv head) pairs of one case: [8, 131072]
    if path == "pages":
        B = _log_int(rng, 1, 16)
        return {"path": path, "B": B, "n_kv": n_kv, "group": group, "S": _log_int(rng, 16, min(131072, most // (B * n_kv)))}
    if path == "slots":
        B = _log_int(rng, 1, 64)
        hi = _log_int(rng, 64, min(32768, most // (B * n_kv)))
        return {"path": path, "B": B, "pad": rng.choice((0, 0, 1, 3)), "n_kv": n_kv, "group": group, "lo": rng.randint(1, hi), "hi": hi, "own": rng.random() < 0.5}
    if path == "paged":
        B, wide = _log_int(rng, 1, 32), rng.random() < 0.3
        hi = _log_int(rng, 64, min(65536, most // (B * n_kv * (2 if wide else 1))))
        return {"path": path, "B": B, "n_kv": n_kv, "group": group, "lo": rng.randint(1, hi), "hi": hi, "wide": wide}
    if path in ("encode", "decode"):
        return {"path": path, "n_kv": n_kv, "S": _log_int(rng, 16, 524288 // n_kv)}
    if path == "prefill":
        B = _log_int(rng, 1, 8)
        return {"path": path, "B": B, "n_kv": n_kv, "L": _log_int(rng, 16, 262144 // (n_kv * B)), "own": rng.random() < 0.5}
    return {"path": path, "n_kv": n_kv, "context": 16 * _log_int(rng, 1, 2048), "new": _log_int(rng, 1, 8192)}


def _lengths(case):
    """Tokens of each sequence before the step, from the case alone: spread between lo and hi, the ends of a block as likely as its middle."""
    r = random.Random("%(B)d %(lo)d %(hi)d" % case)
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["B"])]


def work(case):
    p, n = case["path"], case["n_kv"]
    if p in ("pages", "slots", "paged"):
        lens = [case["S"]] * case["B"] if p == "pages" else [x + 1 for x in _lengths(case)]
        halves = 2 if case.get("wide") else 1
        n_q = n * case["group"]
        part = 0 if p == "pages" else sum(x % T for x in lens)                  # rows of the block that is still filling
        kv = 2 * n * halves * ((sum(lens) - part) * COMPRESSED + part * PLAIN)
        return {"bytes": kv + 2 * len(lens) * n_q * halves * PLAIN, "flops": 4.0 * D * halves * n_q * sum(lens)}
    if p in ("encode", "decode"):
        return {"bytes": 2 * n * case["S"] * (PLAIN + COMPRESSED + (4 if p == "encode" else 0)), "flops": 0}
    if p == "prefill":
        return {"bytes": 2 * n * case["B"] * case["L"] * (PLAIN + COMPRESSED), "flops": 0}
    return {"bytes": 2 * n * (case["context"] + case["new"]) * (PLAIN + COMPRESSED), "flops": 0}


def tolerance(case):
    # attention: BF16 results (2^-8 between neighbours) of fp32 sums; everything else of the format is bit-exact
    return {"rel": 4e-3, "max": 1e-2} if case["path"] in ("pages", "slots", "paged") else "exact"


# ---------------------------------------------------------------------------------------------------------------- state
def _kv(kind, heads, tokens, seed):
    return synth_kv(kind, heads, tokens, seed, "cuda", chunk=max(4096, (1 << 20) // heads))


def _rows(x):
    """[heads, tokens, 128] -> the token-major rows that a model produces."""
    return x.transpose(0, 1).contiguous()


def _queries(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)


def _bases(k, v):
    n = k.shape[0]
    ck, cv = Codec(n).calibrate(k[:, :2048]), Codec(n).calibrate(v[:, :2048])
    return {"k3": ck.base3, "k4": ck.base4, "v3": cv.base3, "v4": cv.base4}


def _sequences(x, B):
    """[n_kv, B * S, 128] -> the heads of B sequences with the same channel scales, [B * n_kv, S, 128]."""
    n = x.shape[0]
    return x if B == 1 else x.view(n, B, -1, D).transpose(0, 1).reshape(B * n, -1, D)


def _prepare_slots(case, seed):
    n, B = case["n_kv"], case["B"]
    lens = _lengths(case)
    k, v = _rows(_kv("k", n, sum(lens) + B, seed)), _rows(_kv("v", n, sum(lens) + B, seed))
    cache = CompressedKVCache(B, n, max(1024, case["hi"] + 64), bases=None if case["own"] else _bases(k[:2048].transpose(0, 1), v[:2048].transpose(0, 1)))
    order = random.Random(B).sample(range(B), B)                                # which slot a row has is up to the scheduler
    at = 0
    for slot, length in zip(order, lens):
        cache.prefill(slot, k[at:at + length], v[at:at + length], check=False)
        at += length
    cache.settle_prefills()
    rows = B + case["pad"]
    slots = torch.tensor(order + [-1] * case["pad"], dtype=torch.int32, device="cuda")
    new = torch.zeros(2, rows, n, D, dtype=torch.bfloat16, device="cuda")
    new[0, :B], new[1, :B] = k[at:], v[at:]
    counters = [cache.S, cache.tail_len, cache.k.ovf_used, cache.v.ovf_used]
    return {"cache": cache, "slots": slots, "k": new[0], "v": new[1], "q": _queries((rows, n * case["group"], D), seed), "longest": max(lens) + 1,
            "counters": counters, "before": [t.clone() for t in counters]}


def _layer_state(n_heads, blocks, k, v):
    """Paged layout: the state of one layer and its block buffer, with some blocks to spare and one raw tile in ten."""
    pool = blocks + blocks // 8 + 4
    st = LayerState(pool, n_heads, raw_tiles=pool * 2 * n_heads // 10 + 64 + 64 * n_heads, bases=_bases(k, v), ovf_slot=OVF_SLOT, device="cuda")
    return st, torch.zeros(pool * 2 * n_heads * (OVF_OFF + OVF_SLOT), dtype=torch.uint8, device="cuda"), np.random.default_rng(blocks).permutation(pool).astype(np.int32)


def _entries(blocks, first_row, tokens):
    """Store entries of `tokens` rows, the first of them at the start of a block."""
    t = np.arange(-(-tokens // T), dtype=np.int64)
    return np.stack([blocks[:t.size], first_row + t * T, 0 * t, np.minimum(T, tokens - t * T)], 1).astype(np.int32)


def _freeq(entries, n_heads):
    return torch.empty(entries * 2 * n_heads, dtype=torch.int32, device="cuda")


def _prepare_paged(case, seed):
    n, B, wide = case["n_kv"], case["B"], case["wide"]
    heads = 2 * n if wide else n
    lens = _lengths(case)
    k, v = _kv("k", heads, sum(lens) + B, seed), _kv("v", heads, sum(lens) + B, seed)
    need = [x // T + 1 for x in lens]
    st, buf, perm = _layer_state(heads, sum(need), k, v)
    k, v = _rows(k), _rows(v)
    bt, ent, step, at, used = np.zeros((B, max(need)), np.int32), [], [], 0, 0
    for i, length in enumerate(lens):
        bt[i, :need[i]] = perm[used:used + need[i]]
        ent.append(_entries(bt[i], at, length))
        step.append((bt[i, length // T], i, length % T, 1))
        at, used = at + length, used + need[i]
    ent = np.concatenate(ent)
    st.store(k, v, buf, torch.from_numpy(ent).cuda(), _freeq(len(ent), heads))
    dim = 256 if wide else D
    counters = [st.mt, st.stack, st.top]
    return {"wide": wide, "st": st, "buf": buf, "bt": torch.from_numpy(bt).cuda(), "k": k[at:].clone(), "v": v[at:].clone(), "n_kv": n, "n_q": n * case["group"],
            "ent": torch.tensor(step, dtype=torch.int32, device="cuda"), "freeq": _freeq(B, heads), "lens": torch.tensor([x + 1 for x in lens], dtype=torch.int32, device="cuda"),
            "q": _queries((B, n * case["group"], dim), seed), "out": torch.empty(B, n * case["group"] * dim, dtype=torch.bfloat16, device="cuda"),
            "counters": counters, "before": [t.clone() for t in counters]}


def _prepare_chunk(case, seed):
    n, ctx, new = case["n_kv"], case["context"], case["new"]
    k, v = _kv("k", n, ctx + new, seed), _kv("v", n, ctx + new, seed)
    blocks = ctx // T + -(-new // T)
    st, buf, perm = _layer_state(n, blocks, k, v)
    k, v = _rows(k), _rows(v)
    old = _entries(perm, 0, ctx)
    st.store(k, v, buf, torch.from_numpy(old).cuda(), _freeq(len(old), n))
    ent = _entries(perm[ctx // T:], 0, new)
    pairs = np.stack([old[:, 0], old[:, 1], old[:, 3]], 1)
    scratch = torch.zeros(2, ctx + new, n, D, dtype=torch.bfloat16, device="cuda")
    return {"st": st, "buf": buf, "k": k[ctx:].clone(), "v": v[ctx:].clone(), "ent": torch.from_numpy(ent).cuda(), "freeq": _freeq(len(ent), n),
            "pairs": torch.from_numpy(pairs).cuda(), "sk": scratch[0], "sv": scratch[1]}


def prepare(case, seed):
    p, n = case["path"], case["n_kv"]
    if p == "slots":
        s = _prepare_slots(case, seed)
    elif p == "paged":
        s = _prepare_paged(case, seed)
    elif p == "chunk":
        s = _prepare_chunk(case, seed)
    elif p == "prefill":
        B, L = case["B"], case["L"]
        k, v = _kv("k", n, B * L, seed), _kv("v", n, B * L, seed)
        bases = None if case["own"] else _bases(k, v)
        s = {"cache": CompressedKVCache(B, n, max(1024, L + 64), bases=bases), "k": _rows(k).view(B, L, n, D), "v": _rows(v).view(B, L, n, D)}
    else:
        B = case.get("B", 1)
        k, v = _kv("k", n, B * case["S"], seed), _kv("v", n, B * case["S"], seed)
        ck, cv = Codec(n).calibrate(k[:, :2048]), Codec(n).calibrate(v[:, :2048])
        # how long an escape stream gets depends on the values: the program keeps room for it, 128 bytes per tile
        s = {"k": k, "v": v, "ck": ck, "cv": cv, "room": torch.zeros(2, n * -(-case["S"] // T) * 128 + 1288, dtype=torch.uint8, device="cuda")}
        if p != "encode":
            s = {"kp": ck.encode(_sequences(k, B), "k"), "vp": cv.encode(_sequences(v, B), "v")}
        if p == "pages":
            s["q"] = _queries((case["B"], n * case["group"], D), seed)
    s["path"] = p
    return s


# ---------------------------------------------------------------------------------------------------------------- one pass
def _page_bytes(pg, room):
    room[:pg.ovf.numel()].copy_(pg.ovf)
    return [pg.sm, pg.codes, pg.flags, pg.ovf_off, room, pg.ovf_head_start, pg.tile_off]


def _cache_bytes(cache):
    return [cache.S, cache.tail_len] + [t for st in (cache.k, cache.v) for t in (st.sm, st.codes, st.flags, st.tile_off, st.ovf, st.ovf_used, st.tail, st.base3, st.base4)]


def run(s):
    p = s["path"]
    if p == "pages":
        return attention(s["q"], s["kp"], s["vp"])
    if p == "slots":
        torch._foreach_copy_(s["counters"], s["before"])
        cache = s["cache"]
        cache.append(s["slots"], s["k"], s["v"])
        return [cache.attention(s["q"], s["slots"], SCALE, max_len=s["longest"])] + _cache_bytes(cache)
    if p == "paged":
        torch._foreach_copy_(s["counters"], s["before"])
        st, attend = s["st"], paged_attention256 if s["wide"] else paged_attention
        st.store(s["k"], s["v"], s["buf"], s["ent"], s["freeq"])
        attend(s["q"], s["out"], s["buf"], st.raw, st.mt, s["bt"], s["lens"], st.bases, st.TS, s["n_q"], s["n_kv"])
        return [s["out"], s["buf"], st.top, st.err]             # which raw tile a block has is free, so the pool and the mode table are not comparable
    if p == "encode":
        return _page_bytes(s["ck"].encode(s["k"], "k"), s["room"][0]) + _page_bytes(s["cv"].encode(s["v"], "v"), s["room"][1])
    if p == "decode":
        return [Codec.decode(s["kp"]), Codec.decode(s["vp"])]
    if p == "prefill":
        cache = s["cache"]
        for slot in range(s["k"].shape[0]):
            cache.prefill(slot, s["k"][slot], s["v"][slot], check=False)
        cache.settle_prefills()
        return _cache_bytes(cache)
    st = s["st"]
    st.decode_blocks(s["buf"], s["pairs"], s["sk"], s["sv"])
    st.store(s["k"], s["v"], s["buf"], s["ent"], s["freeq"])
    return [s["sk"], s["sv"], s["buf"], st.top, st.err]
