"""Fused decode attention over the compressed KV (head_dim 128, GQA group size 1..8) on the B200 CUDA library.

Mirror of gaac/kernel.py: `attention(q, kp, vp, scale, nsplit)` over two Pages, `choose_nsplit`, and `_ext()` whose
`gaac_attn_launch` keeps the argument list of the reference launcher (gaac/kernel.py:296-300) so callers written against the
reference (its slot cache) work unchanged.  One kernel launch does split-K flash decoding over compressed tiles, the raw BF16
tail and the merge of the splits.
"""
from __future__ import annotations
import functools
import torch
from . import _lib

_WS = {}        # (device index, stream, 0) -> workspaces, the last one in use.  Zeroed once: every call leaves its split counters at zero and the header
                # in front of the partials has a fixed size for B*n_q up to 16320, so calls of any such shape share one.  Above that the header
                # depends on B*n_q, which then stands in the key.
SM_COUNT_B200 = 148
ATT_WARPS = 16  # warps per CTA of the CUDA kernel (one CTA per SM)


@functools.lru_cache(maxsize=4096)
def _workspace_bytes(B: int, n_q: int, nsplit: int) -> int:
    return _lib.lib().gaac_attn_workspace_bytes(B, n_q, nsplit)


def workspace(dev, B: int, n_q: int, nsplit: int, stream: int | None = None) -> torch.Tensor:
    """The workspace of the current stream.  One that became too small is kept beside its successor: a captured CUDA graph may hold its address, and the
    successor has at least twice its size, so all of them together stay below twice the largest.  stream: the current stream, where the caller knows it."""
    need = _workspace_bytes(B, n_q, nsplit)
    if not isinstance(dev, torch.device): dev = torch.device(dev)
    key = (dev.index, _lib.stream_ptr(dev) if stream is None else stream, B * n_q if B * n_q > 16320 else 0)
    held = _WS.get(key)
    if held is None:
        held = _WS.setdefault(key, [])
    if not held or held[-1].numel() < need:
        held.append(torch.zeros(max(need, 2 * held[-1].numel() if held else 1 << 20), dtype=torch.uint8, device=dev))
    return held[-1]


def workspace_error(dev, B: int = 0, n_q: int = 0) -> bool:
    """True when a kernel that used a cached workspace of the current stream gave up on a bounded wait for its own asynchronous
    copies (the int32 at the start of the workspace).  Reads device memory, so it synchronises; meant for tests and debugging."""
    here = (torch.device(dev).index, torch.cuda.current_stream(dev).cuda_stream)
    return any(ws[0:4].view(torch.int32).item() != 0 for key, held in _WS.items() if key[:2] == here for ws in held)


def choose_nsplit(B: int, n_kv: int, S: int, target_ctas: int = 96, min_tok: int = 512, cap: int = 48) -> int:
    """Splits per (row, kv head), the reference's heuristic verbatim (gaac/kernel.py:340-342; tuned for a 48-SM GB10)."""
    return min(max(1, target_ctas // (B * n_kv)), max(1, S // min_tok), cap)


@functools.lru_cache(maxsize=4096)
def choose_nsplit_sm100(B: int, n_kv: int, S: int, sm_count: int = SM_COUNT_B200, min_tiles_per_warp: int = 2, ragged: bool = False,
                        total_tokens: int | None = None, teams: bool = True, bound: bool = False) -> int:
    """Splits per (row, kv head) for a B200.  The kernel runs one 16-warp CTA per SM.

    Equal lengths (S is every row's length): the split count minimises a cost model fitted to measurements,
        waves x ((tiles per warp + 0.5) x tile time + per-CTA fixed cost),   waves = ceil(rows x splits / SMs),
    over the counts that leave every warp at least min_tiles_per_warp 16-token tiles (fewer on short contexts, see the code).  Tile time: 4.5 us, 5.2 us
    beyond 512 tiles of a range; fixed cost (prologue, warp merge, split merge): 10 us.  These were fitted to an earlier kernel (the present one takes about
    6.5 us + 0.22 us per tile and CTA, and nothing changes at 512); the counts they choose were not refitted.  Few rows end up with one wave that
    fills the SMs, many rows with ranges of at most 512 tiles in several waves.
    Ragged lengths (ragged=True, S is the longest row; total_tokens is accepted and unused): every row gets the same split count;
    see the comment in the code."""
    rows = max(1, B * n_kv)
    ntiles = max(1, (S + 15) // 16)
    most = max(1, ntiles // (ATT_WARPS * min_tiles_per_warp))
    if ragged and B > 1 and not _short_ranges(rows, ntiles, sm_count):
        # CTAs are handed out longest row first, so the end of the launch is filled by the small ones and what remains is a
        # trade between the per-CTA fixed cost (grows with the split count) and the last chunks of the longest row (shrink with
        # it): the measured optimum follows sqrt(1.8 x longest row's tiles / rows).  Near it, a count whose CTAs fill whole waves
        # is preferred while the launch is only a few waves long.
        star = (1.8 * ntiles / rows) ** 0.5
        lo, hi = max(1, -(-ntiles // 512)), max(most, 1)
        first = min(max(lo, int(0.6 * star)), hi)
        last = max(first, min(hi, int(1.5 * star) + 1))
        def waste(ns):
            w = rows * ns / sm_count
            return 0.0 if w >= 4 else 1.0 - w / -(-w // 1)
        return min(range(first, last + 1), key=lambda ns: (waste(ns) > 0.1, abs(ns - star)))
    # Short contexts: when two tiles per warp would leave more than a quarter of the SMs idle, ranges go below that.  A CTA takes about 6.5 us +
    # 0.215 us per tile (8.3 us at least, with the merge of the splits) and 4.5 us + 0.21 us per tile without splits, so up to 16 tiles one CTA is
    # faster; beyond, splits pay down to four tiles each until there are 16 (one per warp of the merge), more only with 16 tiles each.  Batch 1, 8
    # kv heads: 500 tokens 10.8 -> 8.4 us, 1000: 18.1 -> 8.3, 2000: 15.6 -> 8.8; 4 rows of 1000: 18.6 -> 9.9; 1 kv head, 8000 tokens: 16.3 in 15
    # splits, 13.3 in 32, 17.4 in 125.  A second wave costs more than it shortens (4 rows of 1000 in 6 splits: 15.3).
    # Up to eight ranges of a row are a team (clusters whose partials do not go through global memory), where all teams fit the GPU at a time; there three tiles are enough for a range, and 13 tiles for
    # a second one: batch 1, 8 kv heads, 250 tokens 6.7 -> 6.1, 500 7.2 -> 6.1, 1000 7.8 (15 splits) -> 6.8, 1500 8.2 -> 7.4, 2000 8.0 -> 8.05;  2 rows: 500 8.4 (8 splits) -> 7.2 (6), 1000 9.0 (9) -> 8.0;
    # ten tiles, in three ranges, 5.7 -> 6.2, and 6.8 -> 7.6 with groups of 8.
    # bound=True: S is no more than a bound, the lengths are read on the GPU, where a row of up to 16 tiles takes one CTA whatever the count (fewer_ranges in gaac_attn.cu), and a cluster with
    # nothing to merge costs 0.2 to 0.6 us: 8 kv heads, slots, 12 tiles 6.3 (one CTA), 6.8 (a team), paged 16 tiles 6.9 and 7.4.  The same is lost where the bound is longer and the rows are not (40 x 1
    # of 7 tiles in a table of 28 5.9 -> 6.1), against 7.1 for 9.4 where they are.
    # teams=False: for launches that cannot be one, partials and exchanges.  There the ranges' partials go through global memory all the same: partials of 8 heads, 129 tokens 5.5 (one CTA), 7.1 in three
    # ranges; 256 7.0 and 7.4 in five; 1500 7.6 in 16 and 8.2 in 8; 1700 7.6 and 8.8.
    wave, team = sm_count // rows, _team(rows, True) if teams else 1
    if team > 1 and (ATT_WARPS if bound or team < 6 else 12) < ntiles <= 14 * team:         # (many rows of one CTA each: 32 x 1 of 200 tokens 8.4 -> 8.2 where they are that long, 5.3 -> 5.9 where that is a bound)
        return min(team, ntiles // 3)
    if wave > 1 and 4 * most <= 3 * wave:
        return 1 if ntiles <= ATT_WARPS else min(wave, max(min(16, ntiles // 4), -(-ntiles // 16)))
    tile_us, tile_far_us, fixed_us, staged = 4.5, 5.2, 10.0, 512
    best, best_t = 1, None
    for ns in range(1, min(most, 2 * sm_count) + 1):
        chunk = -(-ntiles // ns)
        waves = -(-rows * ns // sm_count)
        near, far = min(chunk, staged), max(0, chunk - staged)
        t = waves * (near / ATT_WARPS * tile_us + far / ATT_WARPS * tile_far_us + 0.5 * tile_us + fixed_us)   # tiles are handed out on demand: warps end half a tile apart
        if best_t is None or t < best_t * 0.985:                       # prefer fewer splits unless clearly better
            best, best_t = ns, t
    return best


TEAMS = {8: 15, 6: 22, 5: 26, 4: 33, 3: 45, 2: 74}       # ranges of a team: how many teams a B200 has room for (the library asks, and does without them where there are fewer)


def _team(rows: int, spare: bool = False) -> int:
    """Most ranges that a row's team may have when all rows have one.  spare: as the library takes it, which wants room for two more teams of 3 or 5 (see team_ok in gaac_attn.cu)."""
    return next((n for n in TEAMS if rows + (2 if spare and n in (3, 5) else 0) <= TEAMS[n]), 1)


def _short_ranges(rows: int, ntiles: int, sm_count: int = SM_COUNT_B200) -> bool:
    """One wave of CTAs, every row split alike, leaves none of them more than a tile per warp: then it hardly matters which row is the longest, and a plain grid, which plans nothing,
    is the faster launch.  us, shares of units -> this, rows of hi / 8 to hi tokens (B x kv heads):  paged 2 x 8 of 300 8.1 -> 7.0;  8 x 8 of 160 8.5 -> 6.1;  16 x 4 of 500 9.1 -> 8.7;  8 x 4 of
    1100 9.4 -> 8.9;  slots 8 x 8 of 500 10.0 -> 9.0;  32 x 1 of 500 9.2 -> 7.9.  With 17 tiles in the longest row's ranges a warp takes a second one: 2 x 8 of
    2448 tokens 9.4 by shares, 10.4 as a grid, 8 x 2 of 2448 9.0 and 10.2, with one query head 8.2 and 9.8; of 2304 (16 tiles) 9.3 and 9.2,
    9.1 and 9.0, 8.2 and 8.8.  Longer ranges are as fast or faster by shares (3 x 8 of 2000, 21 tiles: 10.3 and 10.2; 16 x 1 of 4000, 28 tiles: 10.2 and 10.9)."""
    return ntiles <= ATT_WARPS * (sm_count // rows) and rows <= sm_count


@functools.lru_cache(maxsize=4096)
def choose_units(B: int, n_kv: int, S: int, sm_count: int = SM_COUNT_B200) -> int:
    """Ranges per kv head that the rows of a ragged batch share by their lengths (S: tokens of the longest), or 0 where every row is split alike
    (choose_nsplit_sm100).  One wave over the SMs, for at most 32 rows (one per lane of the warp that shares them out) and ranges of at least four tiles.
    Rounding to whole ranges costs a share of rows / units, so there must be room for two per row, and for four where rows are long and the several
    waves of the other form cost little beside that.  us per call, other form -> this one (B, kv heads, tokens):  slots 8, 8, 200..3000: 27.3 -> 19.5;
    17, 4, 500..6000: 55.0 -> 36.9;  paged 5, 8, 40..1500: 17.4 -> 11.5;  9, 8, 200..4000: 30.2 -> 27.7;  3, 8, 1000..30000: 53.6 -> 48.0;
    8, 2, 500..30000: 44.3 -> 28.6;  but 8, 8, 4000..40000 (2.25 units per row): 160 -> 180.
    Rows of equal length can leave up to a third of a wave idle where there are two or three units per row (7 rows of 18 units: 2 each).  Where two
    waves of shorter ranges would then be faster by 8 %, the units are those of two waves, and the kernel, which sees the lengths, decides; a CTA
    takes about 8.7 us + 0.22 us per tile here.  One wave -> this:  slots 7, 8, 16000 each: 119.1 -> 108.6;  13, 4, 12000 each: 92.4 -> 86.1;  7, 8,
    8000..16000: 92.4 -> 92.4;  but up to 3 us for CTAs that find nothing to do where few rows are long (13, 4, 2400 and one of 16000: 27.0 -> 30.3)."""
    units, two = sm_count // n_kv, 2 * sm_count // n_kv
    if B > 1 and _short_ranges(B * n_kv, -(-S // 16), sm_count):
        return 0
    if not 2 <= B <= 32 or units < (2 if S <= 16384 else 4) * B:
        return 0
    tiles = -(-S // 16)
    if units < 4 * B and 1.08 * 2 * (8.7 + 0.22 * -(-tiles // (two // B))) < 8.7 + 0.22 * -(-tiles // (units // B)):
        units = two
    return min(units, B * -(-max(S, 1) // 64))


def _flat_line(rows: int, most: int) -> bool:
    """The places of a flat launch's line are counted in 32 bits, and the library refuses one that could be longer.  It goes by what a row MAY hold (`most` tokens: the capacity
    of a slot, the row stride of a block table), not by what the caller says the longest row has."""
    return rows * (-(-most // 16) + 64) < 1 << 30


@functools.lru_cache(maxsize=4096)
def choose_flat(B: int, n_kv: int, S: int, nsplit: int, units: int, group: int = 4, most: int = 0, sm_count: int = SM_COUNT_B200) -> int:
    """CTAs of a flat launch (one wave that shares the tiles of all rows and kv heads evenly), or 0 where the form that it would replace is no slower: nsplit splits per
    (row, kv head), or `units` ranges per kv head (S: tokens that the longest row may have, group: query heads per kv head, most: tokens that any row may hold; nsplit itself
    does not enter).  S is often a bound far above the rows' lengths (a block table as wide as the longest sequence allowed, a cache's capacity): the launch reads the
    lengths and plans accordingly, the grid's split count cannot.
    A flat launch saves what comes with the waves of a grid, and the idle end of the last one; it pays some 8 us for every piece of a row that a CTA has beyond its
    first.  us, other form -> flat:
      grids of several waves: 64 rows x 1 kv head, 32K tokens 219 -> 202;  16 x 8, 4K-64K 452 -> 403;  40 x 4, 2K-6K 98 -> 76;  20 x 8, 2K-3K 68 -> 54;  64 x 8, 500-4200 162 -> 143.
        Short rows in a table that fits them are even: 64 x 8, 100-400 31.6 -> 32.0;  32 x 8, 20-2000 41 -> 42;  24 x 8, 64-600 16.4 -> 16.8;  in one of 8192 tokens they take 57, 68 and 32 as
        a grid
      one wave: 64 x 2, 4K-8K 98 -> 86;  64 x 1, 8K-16K 113 -> 87;  37 x 4, 8K each, paged 118 -> 108, slots 105.5 -> 108.1
      shares of units, which come in whole ones: a fifth of them or more for the rows' first units 8 x 8, 4K-16K 89 -> 77;  4 x 8, 20K-32K 99 -> 91;  5 x 8, 1K-9K 25.3 -> 25.9;  short rows
        there pay for the plan (8 x 8, 200-3000 14.9 -> 15.6);  fewer, 16 x 1 24.6 -> 25.4, 8 x 1 24.8 -> 26.2;  more than four query heads per kv head, 6 x 8 37.6 -> 38.1."""
    rows, tiles = B * n_kv, -(-S // 16)
    if B <= 1 or tiles < 160 or rows * tiles < 120 * sm_count or not _flat_line(rows, max(S, most)):
        return 0
    if units:
        return sm_count if group <= 4 and 5 * B >= units else 0
    return sm_count


@functools.lru_cache(maxsize=4096)
def choose_flat256(B: int, n_kv: int, S: int, most: int = 0, sm_count: int = SM_COUNT_B200, group: int = 4) -> int:
    """The same for head_dim 256, whose grid hands the rows out as they come.  us, grid -> flat: 8 rows x 4 kv heads, 1K-8K tokens 33.1 -> 24.8;  20 x 8, up to 3K 95 -> 73;  32 x 2, up
    to 4K 56 -> 40;  6 x 2, up to 60K 124 -> 93;  8 x 4, 100-700 22.0 -> 13.2;  2 x 8 of 1000 30 -> 13;  9 x 4, up to 1500 23.8 -> 16.6;  30 x 4, up to 2K 55 -> 48;  32 x 4, up to 1000 30.7 -> 31.4,
    in a table of 8192 43 -> 31;  32 x 8 the same 53 -> 40, 65 -> 40.  A full wave of equal rows is the grid's: 12 x 4 of 4000 45.3 -> 47.6;  so are a few very short ones: 4 x 4 of 50-300 in a
    table of 8192 9.4 -> 11.0;  one sequence has nothing to gain: 1 x 4 of 8K 17.9 -> 18.4.
    More rows than SMs: from 160 tiles on, since rows much shorter than the table pay for the plan and for dearer pieces.  20 x 8 in a table of 72 tiles, rows of 18 23.1 -> 23.9 (groups of 8 26.9 ->
    31.2), of 2-18 12.7 -> 14.6;  of 112, rows of 3-28 16.0 -> 17.9;  of 144, rows of 5-36 21.6 -> 20.8;  what rows as long as such a table would gain (70 tiles each 65 -> 47, 9-70 38.5 -> 34.5) is left.
    A wave of equal ranges (_splits256) comes first where a CTA gets no more than 24 tiles, or 16 with groups of up to 4, whose ragged rows are better off by shares: 27 x 2 of 6-48 tiles, two ranges
    each, 16.6, flat 15.2;  40 x 1 of 9-70 in three 16.5 and 15.3;  5 x 4 of 19-150 in seven 16.6 and 15.9;  groups of 8 20.1 and 19.9, 19.9 and 19.7, 20.4 and 20.5."""
    rows, tiles = B * n_kv, -(-S // 16)
    if B <= 1 or not _flat_line(rows, max(S, most)) or tiles < (48 if 2 * rows <= sm_count else 96 if rows <= sm_count else 160):
        return 0
    ns = _splits256(rows, tiles, group, sm_count)
    return 0 if ns and tiles <= (16 if group <= 4 else 24) * ns else sm_count


def _splits256(rows: int, tiles: int, group: int = 4, sm_count: int = SM_COUNT_B200) -> int:
    """Splits of one wave in which every row is split alike, where that leaves a CTA at most three tiles per pair of its warps, or 0.  Ranges of four tiles until there are 16 of them, then of
    eight (a tile per pair) until there are 32: us, one row, groups of 4 and 8, by the number of ranges:  70 tiles 16: 9.9 and 13.7, 17: 10.4 and 14.3;  150 tiles 16: 12.5 and 16.3, 19: 11.5 and 15.1,
    37: 11.5 and 15.6;  250 tiles 32: 12.2 and 16.0, 62: 12.5 and 16.2;  600 tiles 32: 17.0 and 21.1, 74: 18.8 and 25.6.  More than 16 want to save a turn of the pairs: 8 heads x 150 tiles 16: 13.1 and
    16.7, 18: 13.3 and 17.3.  With groups of 5 to 8 the merge is dearer: 16 tiles stay in one CTA (27 x 2 of 10 tiles 11.3, in two ranges 12.8;  1 x 8 of 9 10.7, in three 12.4;  40 x 1 of 18 14.4
    and 13.3), 24 where a row could only have two (27 x 2 of 18 tiles 14.4 and 15.5, of 28 17.9 and 16.5)."""
    wave = sm_count // rows if rows <= sm_count else 1
    ns = min(wave, max(1, min(8, tiles // 3), min(16, tiles // 4), min(32, -(-tiles // 8))))
    if 16 < ns and 8 * ns < tiles <= 256: ns = 16
    if tiles <= (8 if group <= 4 else 24 if ns == 2 else 16): ns = 1               # (as fewer_ranges in gaac_attn.cu)
    return ns if wave > 1 and tiles <= 24 * ns else 0


@functools.lru_cache(maxsize=4096)
def choose_nsplit256(B: int, n_kv: int, S: int, sm_count: int = SM_COUNT_B200, group: int = 4) -> int:
    """Splits per (row, kv head) at head_dim 256, whose CTAs work on eight tiles at a time.  S may be a bound far above the rows' lengths: the kernel takes fewer ranges for a row of few
    tiles.  One wave of short ranges comes first; us, the counts made for 16 warps, or a flat launch, -> this, rows of hi / 8 to hi tokens (B x kv heads): 2 x 1 of 740 17.3 -> 8.9;  8 x 4 of 500 16.0 -> 10.8;
    5 x 8 of 740 20.9 -> 13.5;  2 x 4 of 4000 15.8 (flat) -> 13.7;  8 x 8 of 1100 20.8 (flat) -> 19.2;  1 x 1 of 300 10.2 -> 8.2."""
    return _splits256(B * n_kv, -(-S // 16), group, sm_count) or choose_nsplit_sm100(B, n_kv, S, ragged=True, teams=False)


def _flat_splits(B: int, n_kv: int, ctas: int) -> int:
    return 1 + -(-ctas // (B * n_kv))            # what the workspace must have room for


def _side(sm, codes, flags, tile_off, ovf, head_start, base3, base4, tail) -> _lib.Side:
    return _lib.Side(sm.data_ptr(), codes.data_ptr(), flags.data_ptr(), tile_off.data_ptr(), ovf.data_ptr(), head_start.data_ptr(),
                     ovf.numel(), base3.data_ptr(), base4.data_ptr(), _lib.ptr(tail))


class _Ext:
    """Stand-in for the reference's JIT-built extension module."""

    @staticmethod
    def gaac_attn_launch(smk, ck, fk, tok, ovk, ohsk, b3k, b4k, smv, cv, fv, tov, ovv, ohsv, b3v, b4v,
                         q, slot, n_q, n_kv, SL, S_pad, scale, nsplit, kt, vt, TL, TCAP, out_f32=None, partial=None, exchange=None, fused=False, units=0, flat=0):
        """Same positional arguments as the reference launcher (gaac/kernel.py:296-300): 16 K/V buffers, q [B*n_q, 128] bf16,
        slot int32 [B], n_q, n_kv, SL int32 [heads], S_pad, scale, nsplit, K/V tails [heads, TCAP, 128] bf16 (empty = none),
        TL int32 [heads], TCAP.  Returns out [B*n_q, 128] bf16.  Extras: out_f32 (fp32 tensor to receive the un-rounded
        result), partial ([B*n_q, 130] fp32 tensor: write (m, l, acc) there instead of the output), exchange (a
        gaac_b200._lib.Exchange: push the partial rows into every rank's receive buffer instead and return None; with fused=True
        the same launch also waits for the other ranks' rows, merges them and returns the output), units (> 0: the rows share that many
        ranges per kv head by their lengths, nsplit is not used), flat (> 0: one wave of that many CTAs, see choose_flat)."""
        D = 128
        if q.size(-1) != D:
            raise RuntimeError("head_dim must be 128")
        G = n_q // max(1, n_kv)
        if not (1 <= G <= 8 and G * n_kv == n_q):
            raise RuntimeError("GQA group size must be 1..8")
        if not q.is_cuda:
            raise RuntimeError("gaac_b200 attention needs CUDA tensors: there is no CPU path")
        dev = q.device
        B = slot.size(0)
        has_tail = kt.numel() > 0
        stream = _lib.stream_ptr(dev)
        ws = workspace(dev, B, n_q, _flat_splits(B, n_kv, flat) if flat else -(-units // B) if units else nsplit, stream)
        if exchange is None and partial is None:
            H = _lib.host()
            out = H.empty(q, 3, B * n_q, D) if isinstance(q, torch.Tensor) else torch.empty(B * n_q, D, dtype=q.dtype, device=dev)
            name = "gaac_decode_attn_flat" if flat else "gaac_decode_attn_balanced" if units else "gaac_decode_attn"
            _lib.check(getattr(H, name)((smk, ck, fk, tok, ovk, ohsk, b3k, b4k, kt if has_tail else None), (smv, cv, fv, tov, ovv, ohsv, b3v, b4v, vt if has_tail else None),
                                        q.data_ptr(), slot, B, n_q, n_kv, SL, S_pad, float(scale), flat or units or int(nsplit), TL if has_tail else None, int(TCAP) if has_tail else 0,
                                        b3k.size(0), ws, ws.numel(), out, out_f32, stream), name)
            return out
        L = _lib.lib()
        K = _side(smk, ck, fk, tok, ovk, ohsk, b3k, b4k, kt if has_tail else None)
        V = _side(smv, cv, fv, tov, ovv, ohsv, b3v, b4v, vt if has_tail else None)
        common = (K, V, q.data_ptr(), slot.data_ptr(), B, n_q, n_kv, SL.data_ptr(), S_pad, float(scale), int(nsplit),
                  TL.data_ptr() if has_tail else None, int(TCAP) if has_tail else 0, b3k.size(0), ws.data_ptr(), ws.numel())
        if exchange is not None and fused:
            out = torch.empty(B * n_q, D, dtype=q.dtype, device=dev)
            _lib.check(L.gaac_decode_attn_exchange(*common, exchange, out.data_ptr(), _lib.ptr(out_f32), stream), "gaac_decode_attn_exchange")
            return out
        if exchange is not None:
            _lib.check(L.gaac_decode_attn_push(*common, exchange, stream), "gaac_decode_attn_push")
            return None
        _lib.check(L.gaac_decode_attn_partial(*common, partial.data_ptr(), stream), "gaac_decode_attn_partial")
        return partial


_mod = None


def _ext():
    global _mod
    if _mod is None:
        _lib.lib()          # fail now, loudly, when the library has not been built
        _mod = _Ext()
    return _mod


def attention(q, kp, vp, scale=None, nsplit=None, out_f32=None, out=None):
    """Decode attention over two Pages (kinds 'k' / 'v', H = B*n_kv heads of equal length).
    q: [B, n_q, D] bf16 (one query token per sequence) -> [B, n_q, D] bf16.  (gaac/kernel.py:345-359)
    out (contiguous bf16 tensor of B*n_q*D elements) receives the result instead of a new tensor; out_f32 (fp32, same shape)
    additionally receives the result before its rounding to BF16.
    nsplit=None picks the B200 heuristic; an explicit nsplit is honoured as given.  us a call over 500 tokens, through ctypes and descriptors kept on the
    Pages -> the native module, which reads the Pages: 10.7 -> 7.3 (the launch takes 5.8 in a graph; what is left above it is this function)."""
    B, n_q, Dq = q.shape
    if Dq != 128:
        raise RuntimeError("head_dim must be 128")
    if not q.is_cuda:
        raise RuntimeError("gaac_b200 attention needs CUDA tensors: there is no CPU path")
    n_kv = kp.H // B
    G = n_q // max(1, n_kv)
    if not (1 <= G <= 8 and G * n_kv == n_q):
        raise RuntimeError("GQA group size must be 1..8")
    if nsplit is None: nsplit = choose_nsplit_sm100(B, n_kv, kp.S)
    if out is None:
        out = _lib.host().empty(q, 3, B, n_q, Dq)
    elif out.is_contiguous() and out.dtype == q.dtype and out.numel() == B * n_q * Dq:
        out = out.view(B, n_q, Dq)
    else:
        raise RuntimeError("out must be a contiguous bf16 tensor with B*n_q*128 elements")
    _pages_call(q, kp, vp, B, n_q, n_kv, scale, nsplit, out=out, out_f32=out_f32)
    return out


def _page_side(pg) -> _lib.Side:
    """The gaac_side descriptor of a Page for ctypes calls (an exchange, a Page without tokens), built once and kept on the Page object (rebuilt when its escape stream was replaced)."""
    sd = getattr(pg, "_attn_side", None)
    if pg.S == 0:                                  # a Page without tokens (a rank past the end of a short context): nothing is read through
        if sd is None:                             # these pointers, but the library wants them non-null, so they point at a small zero buffer
            z = torch.zeros(256, dtype=torch.uint8, device=pg.base3.device)
            sd = _side(z, z, z, z, z, pg.ovf_head_start, pg.base3, pg.base4, None)
            pg._attn_side, pg._attn_keep = sd, z
        return sd
    if sd is None or sd.ovf != pg.ovf.data_ptr() or sd.sm != pg.sm.data_ptr():
        sd = _side(pg.sm, pg.codes, pg.flags, pg.tile_off, pg.ovf, pg.ovf_head_start, pg.base3, pg.base4, None)
        pg._attn_side = sd
    return sd


def _pages_call(q, kp, vp, B, n_q, n_kv, scale, nsplit, out=None, out_f32=None, part=None, exchange=None, fused=False):
    """One gaac_decode_attn_pages call: every head of the two Pages holds kp.S tokens and batch row b reads heads b*n_kv ..,
    which is all the identity slot map and the constant length table of the reference's entry point said
    (gaac/kernel.py:349-352); the kernel needs neither table."""
    dev = q.device
    if not q.is_contiguous(): q = q.contiguous()
    stream = _lib.stream_ptr(dev)
    ws = workspace(dev, B, n_q, nsplit, stream)
    if exchange is None and kp.S > 0:
        _lib.check(_lib.host().gaac_decode_attn_pages(kp, vp, q, B, n_q, n_kv, kp.S, max(16, kp.sm.shape[1] // 128), float(scale if scale is not None else 128 ** -0.5), int(nsplit),
                                                      kp.base3.size(0), ws, ws.numel(), out, out_f32, part, None, 1 if fused else 0, stream), "gaac_decode_attn_pages")
        return
    _lib.check(_lib.lib().gaac_decode_attn_pages(_page_side(kp), _page_side(vp), q.data_ptr(), B, n_q, n_kv, kp.S, max(16, kp.sm.shape[1] // 128),
                                                 float(scale if scale is not None else 128 ** -0.5), int(nsplit), kp.base3.size(0),
                                                 ws.data_ptr(), ws.numel(), _lib.ptr(out), _lib.ptr(out_f32), _lib.ptr(part), exchange,
                                                 1 if fused else 0, stream), "gaac_decode_attn_pages")


def combine(pm: torch.Tensor, pl: torch.Tensor, pa: torch.Tensor, out_f32: torch.Tensor | None = None) -> torch.Tensor:
    """Merge partials pm, pl [n_heads, n_parts] and pa [n_heads, n_parts, 128] (fp32, m in natural-log units) -> [n_heads, 128] bf16
    (gaac/kernel.py:281-294)."""
    n_heads, n_parts = pm.shape
    out = torch.empty(n_heads, 128, dtype=torch.bfloat16, device=pm.device)
    _lib.check(_lib.lib().gaac_combine(pm.contiguous().data_ptr(), pl.contiguous().data_ptr(), pa.contiguous().data_ptr(), n_heads, n_parts,
                                       out.data_ptr(), _lib.ptr(out_f32), _lib.stream_ptr(pm.device)), "gaac_combine")
    return out


def combine_parts(parts: torch.Tensor, out_f32: torch.Tensor | None = None) -> torch.Tensor:
    """Merge packed partials [n_parts, n_heads, 130] fp32 (rows of (m, l, acc[128]), m in natural-log units) -> [n_heads, 128] bf16:
    the buffer an all-gather of the ranks' partial outputs produces, merged in one launch."""
    n_parts, n_heads, w = parts.shape
    assert w == 130 and parts.is_contiguous()
    out = torch.empty(n_heads, 128, dtype=torch.bfloat16, device=parts.device)
    _lib.check(_lib.lib().gaac_combine_parts(parts.data_ptr(), n_heads, n_parts, out.data_ptr(), _lib.ptr(out_f32), _lib.stream_ptr(parts.device)),
               "gaac_combine_parts")
    return out
