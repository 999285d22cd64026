// Cache maintenance kernels (sm_100a): slot-layout append, paged-layout store / release / block decode.
#include <algorithm>
#include "gaac_api.cuh"
#include "gaac_warp.cuh"

namespace gaac {

// ------------------------------------------------------------------------------------------------ slot layout: append
struct AppendParams {
  gaac_store K, V;
  const uint16_t *k_new, *v_new;
  const int* slot; int n_kv;
  int *tail_len, *seq_len;
  long S_cap, ovf_cap; int n_base_rows;
  int* err;
};

// One CTA per (batch row, kv head): warp 0 appends K, warp 1 appends V; the shared counters are advanced once both are done
// (the reference needs a second launch for that: gaac/kv_cache.py:72-73,87-96).
// Bound by its chain of loads, from the slot number on; the new row travels with the slot number and the bases of a tile that fills with its rows (us, append and attention in a graph: 7 rows of up to
// 3000 tokens 19.35 -> 19.2, 64 of 32768 188.5 -> 187.7).
// First half: the new row goes into the tail; when that fills the tail, the 16 rows are encoded into registers.  Returns the
// tile's escape bytes, or -1 when there is no tile to store (tail not full, or the head is at its token capacity).
template <int KIND_V>
__device__ __forceinline__ int append_encode(WarpScratch& ws, const gaac_store& st, uint2 row, long h, int pos, int tile, long S_cap,
                                             int n_base_rows, int lane, LaneTile& lt) {
  uint16_t* tail = reinterpret_cast<uint16_t*>(st.tail) + h * (T * D);
  reinterpret_cast<uint2*>(tail + (long)pos * D)[lane] = row;                 // 32 lanes x 8 B
  if (pos + 1 != T) return -1;
  if ((long)tile * T + T > S_cap) return -1;          // cache full: never write past the head's capacity (callers check capacity at prefill)
  const int brow = (int)(h % n_base_rows);
  u32 b3w[8], b4w[8];
  load_base_words<KIND_V>(st.base3 + (long)brow * D, st.base4 + (long)brow * D, lane, b3w, b4w);
  __syncwarp();
  stage_rows(ws, tail, D, T, lane);                   // rows written by this warp just now are visible to it after the barrier
  return encode_tile_warp<KIND_V>(ws, T, b3w, b4w, lane, lt);
}
// Second half: the encoded tile goes to the head's streams, its escape bytes behind the bytes in use.
template <int KIND_V>
__device__ __forceinline__ void append_store(WarpScratch& ws, const gaac_store& st, const LaneTile& lt, long h, int tile, int total, long S_cap, long ovf_cap, int lane) {
  const long trow = h * S_cap + (long)tile * T;
  store_tile_payload<KIND_V>(lt, st.sm + trow * D, st.codes + trow * CB, reinterpret_cast<uint8_t*>(st.flags + trow), lane);
  const int used = st.ovf_used[h];
  store_tile_escapes<KIND_V>(ws, lt, st.ovf + h * ovf_cap + used, lane);
  __syncwarp();
  if (lane == 0) { st.tile_off[h * (S_cap / T) + tile] = used; st.ovf_used[h] = used + total; }
}

__global__ void __launch_bounds__(64) append_kv_kernel(const __grid_constant__ AppendParams p) {
  __shared__ __align__(16) WarpScratch scratch[2];
  __shared__ int s_fit[2];
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  griddep_wait();
  griddep_launch();                                   // the step's attention may set up its tables meanwhile
  const int sl = p.slot[i / p.n_kv];
  const uint2 row = reinterpret_cast<const uint2*>((warp == 0 ? p.k_new : p.v_new) + (long)i * D)[lane];          // (travels with the slot number)
  if (sl < 0) return;
  const long h = (long)sl * p.n_kv + i % p.n_kv;
  const int pos = p.tail_len[h], tile = p.seq_len[h] / T;
  LaneTile lt;
  const gaac_store& st = warp == 0 ? p.K : p.V;
  const int total = warp == 0 ? append_encode<0>(scratch[0], p.K, row, h, pos, tile, p.S_cap, p.n_base_rows, lane, lt)
                              : append_encode<1>(scratch[1], p.V, row, h, pos, tile, p.S_cap, p.n_base_rows, lane, lt);
  // A tile whose escape bytes (plus the 8 bytes a reader may touch behind them) do not fit what is left of the head's escape
  // stream is not stored, for K and V alike: nothing is written outside the head's share, the counters stay, *err counts it.
  if (lane == 0) s_fit[warp] = total < 0 || (long)st.ovf_used[h] + total + 8 <= p.ovf_cap;
  __syncthreads();                                    // both warps have read the counters
  const bool fits = s_fit[0] && s_fit[1];
  if (total >= 0 && fits) {
    if (warp == 0) append_store<0>(scratch[0], p.K, lt, h, tile, total, p.S_cap, p.ovf_cap, lane);
    else append_store<1>(scratch[1], p.V, lt, h, tile, total, p.S_cap, p.ovf_cap, lane);
  }
  if (threadIdx.x == 0) {
    const int t = pos + 1, full = (t == T);
    if (full && !fits) { if (p.err) atomicAdd(p.err, 1); return; }
    if (full && (long)tile * T + T > p.S_cap) return;   // cache full: the tile was not stored, keep the counters (the last tail row is overwritten next time)
    p.tail_len[h] = full ? 0 : t;
    if (full) p.seq_len[h] = p.seq_len[h] + T;
  }
}

// ------------------------------------------------------------------------------------------------ paged layout
struct PagedParams {
  gaac_paged st;
  const uint16_t *key, *value; long k_stride, v_stride;
  const int* ent; int* freeq;
};

// -1: the pool is empty, which is counted; top then stays below zero by the failed pops of the step.
__device__ __forceinline__ int pop_raw_tile(const gaac_paged& st, int lane) {
  int r = -1;
  if (lane == 0) {
    const int idx = atomicAdd(st.top, -1) - 1;
    if (idx >= 0) r = st.stack[idx]; else atomicAdd(st.err, 1);
  }
  return __shfl_sync(FULL, r, 0);
}
// No pop is under way (they are in another launch or behind a barrier).  Failed pops took nothing, so a top below zero counts as zero; every
// push sees to that before its own addition, and after the first one top never is below zero again.
__device__ __forceinline__ void push_raw_tile(int* stack, int* top, int r) {
  atomicMax(top, 0);
  stack[atomicAdd(top, 1)] = r;
}

// One warp: entry e, tile slot t = 2*kvh + kind.  Returns (lane 0) the raw tile that the store set free, or -1: it may go back on the stack once no
// warp of the step pops any more.
// Bound by its chain of loads: the entry, the mode table, rows and bases, then the encoder's work.  New rows and bases do not depend on the table and travel with its entry; behind one another
// they cost most where no cache holds them: a step of 8 rows at head_dim 256, store and attention over two states in turn, 38.1 -> 34.5 us (58 MB of slots each); out of L2 32 x 8 blocks that fill
// 9.2 -> 8.1.  (The rows of a block that stays raw wait for its tile: ahead of the entry they gained nothing.)  A block that is new as a whole has no old rows to ask for: asked one by one
// whether they are there, 24 tiles took 4.8 us in place of 4.7 (now 4.6).
template <int KIND_V>
__device__ __forceinline__ int store_one(WarpScratch& ws, const PagedParams& p, int e, int t, int lane) {
  const gaac_paged& st = p.st;
  const int kvh = t >> 1, NT = 2 * st.n_kv;
  const int blk = p.ent[4 * e], tok0 = p.ent[4 * e + 1], off0 = p.ent[4 * e + 2], n = p.ent[4 * e + 3];
  if (blk < 0) return -1;
  const long pt = (long)blk * NT + t;
  const int old = st.mt[pt];
  const bool have = old < 0 && old != ~RAW_NONE, full = (off0 + n == T);       // a block that found the pool empty before asks again
  const int r_old = old < 0 ? raw_tile(old) : 0;
  const uint16_t* src = (KIND_V ? p.value : p.key) + (long)kvh * D;
  const long sstride = KIND_V ? p.v_stride : p.k_stride;
  uint16_t* rawp = reinterpret_cast<uint16_t*>(st.raw);
  int fits = 0, r = r_old;
  // The usual step of a row per block comes first in the code: behind the encoder it took 2.06 us in place of 2.01 (6 x 2 blocks of one row; 2 x 1 whole blocks 3.2 and 3.3).
  const auto keep_raw = [&] {
    if (!have) r = pop_raw_tile(st, lane);
    // new rows, natural channel order, into raw tile r
    for (int c = lane; c < (r < 0 ? 0 : n * 16); c += 32) {
      const int row = off0 + (c >> 4), col = (c & 15) * 8;
      *reinterpret_cast<uint4*>(rawp + ((long)r * T + row) * D + col) = *reinterpret_cast<const uint4*>(src + (long)(tok0 + row - off0) * sstride + col);
    }
  };
  if (!full) keep_raw();
  else {
    // gather the tile: new rows from this step's K/V, which travel with the mode-table entry, old rows from the raw tile (if any)
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int c = lane + 32 * k, row = c >> 4, col = (c & 15) * 8;
      v[k] = make_uint4(0, 0, 0, 0);
      if (row >= off0) v[k] = *reinterpret_cast<const uint4*>(src + (long)(tok0 + row - off0) * sstride + col);
    }
    u32 b3w[8], b4w[8];
    load_base_words<KIND_V>((KIND_V ? st.b3v : st.b3k) + kvh * D, (KIND_V ? st.b4v : st.b4k) + kvh * D, lane, b3w, b4w);
    if (off0 > 0 && have) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int row = (lane >> 4) + 2 * k;
        if (row < off0) v[k] = reinterpret_cast<const uint4*>(rawp + (long)r_old * T * D)[lane + 32 * k];
      }
    }
#pragma unroll
    for (int k = 0; k < 8; k++) *reinterpret_cast<uint4*>(&ws.xs[((lane >> 4) + 2 * k) * XS_STRIDE + (lane & 15) * 8]) = v[k];
    LaneTile lt;
    const int total = encode_tile_warp<KIND_V>(ws, T, b3w, b4w, lane, lt);
    fits = total <= st.ovf_slot;
    if (fits) {
      uint8_t* base = st.buf + pt * st.TS;
      store_tile_payload<KIND_V>(lt, base, base + SLOT_CD_OFF, base + SLOT_FL_OFF, lane);
      store_tile_escapes<KIND_V>(ws, lt, base + SLOT_OVF_OFF, lane);
    }
    if (!fits) keep_raw();
  }
  if (lane == 0) st.mt[pt] = fits ? (int)pt : ~(r < 0 ? RAW_NONE : r);
  return fits && have ? r_old : -1;
}

// 28 CTAs per SM (72 registers): with 80, 25 CTAs, a step of 475 x 8 tiles has a second wave, 7.9 -> 8.9 us.
__global__ void __launch_bounds__(32, 28) paged_store_kernel(const __grid_constant__ PagedParams p) {
  __shared__ __align__(16) WarpScratch ws;
  const int e = blockIdx.x, t = blockIdx.y, lane = threadIdx.x;
  griddep_wait();
  griddep_launch();
  const int freed = t & 1 ? store_one<1>(ws, p, e, t, lane) : store_one<0>(ws, p, e, t, lane);
  if (lane == 0) p.freeq[e * 2 * p.st.n_kv + t] = freed;
}

// The same for a step of few tiles, as ONE cluster: the cluster's barrier stands between the pops and the pushes, so no second launch is needed to
// return the raw tiles.  A warp per tile, 8 blocks (the portable cluster size) of as many warps as 48 KB of static shared memory have room for.  us per
// call, two launches -> this: 16 to 80 tiles 3.0 -> 2.5 where no block completes, 4.2 -> 3.9 where all do.  With 16 warps (128 tiles) steps of 96
// to 128 tiles take 2.8 -> 2.5 and 4.0 -> 4.3, and completing blocks in smaller steps 0.3 more: the warps of an SM share its units while they encode.
constexpr int STEP_WARPS = 11, STEP_CLUSTER = 8;
static_assert(STEP_WARPS * sizeof(WarpScratch) <= 48 * 1024 && (STEP_WARPS + 1) * sizeof(WarpScratch) > 48 * 1024, "");
__global__ void __launch_bounds__(STEP_WARPS * 32) paged_store_step_kernel(const __grid_constant__ PagedParams p, int n_items) {
  __shared__ __align__(16) WarpScratch ws[STEP_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * STEP_WARPS + warp, NT = 2 * p.st.n_kv;
  griddep_wait();
  griddep_launch();
  int freed = -1;
  if (i < n_items) freed = i & 1 ? store_one<1>(ws[warp], p, i / NT, i % NT, lane) : store_one<0>(ws[warp], p, i / NT, i % NT, lane);
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (lane == 0 && freed >= 0) push_raw_tile(p.st.stack, p.st.top, freed);
}

__global__ void __launch_bounds__(256) free_tiles_kernel(const int* __restrict__ freeq, int n_items, int* __restrict__ stack, int* __restrict__ top) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  griddep_wait();
  griddep_launch();
  if (i >= n_items) return;
  const int r = freeq[i];
  if (r >= 0) push_raw_tile(stack, top, r);
}

__global__ void __launch_bounds__(32) release_blocks_kernel(const int* __restrict__ blocks, int NT, int* __restrict__ mt, int* __restrict__ stack, int* __restrict__ top) {
  const long blk = blocks[blockIdx.x];
  for (int t = threadIdx.x; t < NT; t += 32) {
    const long pt = blk * NT + t;
    const int m = mt[pt];
    if (m < 0) { if (m != ~RAW_NONE) push_raw_tile(stack, top, raw_tile(m)); mt[pt] = (int)pt; }
  }
}

// One warp per (entry, tile slot); the CTA's four entries have the slot index t = 2*kvh + kind in common, and with it the tables.
// grid = (ceil(P / 4), 2*n_kv).
// Bound by its chain of loads (entry, mode table, tile, escape bytes behind the tags, then the stores): the first three are asked for before the tables are made.  The tile's place is known without the
// mode table, but asked for together with its entry a raw tile's slot is read for nothing: two states in turn, 384 blocks of 16 tiles 9.7 -> 9.4 us, with one block in ten raw 12.1 -> 12.3, all of them
// 12.6 -> 17.4;  2048 blocks 43.0 -> 42.2, 47.7 -> 48.3 and 56.2 -> 66.2.  384 blocks decoded and 1500 tokens stored: 24.7 -> 24.6 us.  128 bytes of the slot's escape bytes asked for with the tile: 19.0 -> 18.1 with everything in L2,
// but 24.4 and nothing gained from memory, where most of them are not the tile's.  9 CTAs per SM (56 registers, no spills): with 7 (72 registers) the chunk takes 20.9 us, now 20.0, and one behind 32768
// tokens 57.7, now 54.4;  8 20.4 and 55.1;  10 (spills) 22.8 and 67.  All of these with the same blocks again and again, out of L2: where no earlier pass has touched them, the whole chunk (with
// the overlapped launches 24.6 -> 20.4) gains about 1 %.
constexpr int PDEC_WARPS = 4;
// Shared memory's share: 196 KB of an SM's 256, which nine CTAs fit with slots of up to 768 escape bytes and eight with any.  Left to itself the driver makes room for nine, and with 28 KB of L1 the
// codes, which are read 12 bytes apart, do not stay there: slots of 1280 bytes, 2048 blocks 51.0 us, now 44.3 (slots of 128 42.5 as before); with 85 in place of 80 slots of 832 to 960 are left out.
constexpr int PDEC_SHARED = 80;
struct PagedDecodeParams { gaac_paged st; const int* pairs; int P; uint16_t *sk, *sv; long row_stride; };

template <int KIND_V>
__device__ __forceinline__ void decode_blocks_cta(uint8_t* scratch, DecodeTables& tables, const PagedDecodeParams& p, int t) {
  const gaac_paged& st = p.st;
  const int kvh = t >> 1, NT = 2 * st.n_kv, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = blockIdx.x * PDEC_WARPS + warp;
  WarpScratch& ws = *reinterpret_cast<WarpScratch*>(scratch + warp * decode_scratch_bytes(min(st.ovf_slot, TILE_MAX_ESC)));
  griddep_wait();
  griddep_launch();
  // the tile travels while the tables are made
  int row0 = 0, nvalid = 0, m = 0;
  TileWords<KIND_V> tw;
  if (e < p.P) {
    row0 = p.pairs[3 * e + 1]; nvalid = p.pairs[3 * e + 2];
    const long pt = (long)p.pairs[3 * e] * NT + t;
    const uint8_t* base = st.buf + pt * st.TS;
    m = st.mt[pt];
    if (m >= 0) load_tile_words<KIND_V>(tw, base, base + SLOT_CD_OFF, base + SLOT_FL_OFF, base + SLOT_OVF_OFF, 0, lane);
  }
  const u32 w = fill_decode_tables<KIND_V>(tables, (KIND_V ? st.b3v : st.b3k) + kvh * D, (KIND_V ? st.b4v : st.b4k) + kvh * D);
  __syncthreads();
  if (e >= p.P) return;
  uint16_t* dst = (KIND_V ? p.sv : p.sk) + (long)row0 * p.row_stride + (long)kvh * D;
  if (m < 0) {
    const uint16_t* rawp = reinterpret_cast<const uint16_t*>(st.raw) + (long)raw_tile(m) * T * D;
    for (int c = lane; c < nvalid * 16; c += 32) {
      const int row = c >> 4, col = (c & 15) * 8;
      *reinterpret_cast<uint4*>(dst + (long)row * p.row_stride + col) = *reinterpret_cast<const uint4*>(rawp + row * D + col);
    }
    return;
  }
  decode_tile_warp<KIND_V>(ws, tw, w, lane, min(st.ovf_slot, TILE_MAX_ESC));
  unstage_rows(ws, dst, p.row_stride, nvalid, lane);
}
__global__ void __launch_bounds__(PDEC_WARPS * 32, 9) paged_decode_blocks_kernel(const __grid_constant__ PagedDecodeParams p) {
  extern __shared__ __align__(16) uint8_t scratch[];
  __shared__ __align__(16) DecodeTables tables;
  const int t = blockIdx.y;
  if (t & 1) decode_blocks_cta<1>(scratch, tables, p, t); else decode_blocks_cta<0>(scratch, tables, p, t);
}

static int check_paged(const gaac_paged* st) {
  if (!st || !st->buf || !st->raw || !st->mt || !st->stack || !st->top || !st->err || !st->b3k || !st->b4k || !st->b3v || !st->b4v) return GAAC_E_ARG;
  if (st->n_kv <= 0 || st->n_kv > 32767) return GAAC_E_ARG;
  if (st->TS % 16 || st->TS != SLOT_OVF_OFF + st->ovf_slot || st->ovf_slot < 0) return GAAC_E_UNSUPPORTED;
  if (!aligned16(st->buf) || !aligned16(st->raw)) return GAAC_E_ALIGN;
  return GAAC_OK;
}

}  // namespace gaac

using namespace gaac;

extern "C" int gaac_append_kv(const gaac_store* K, const gaac_store* V, const void* k_new, const void* v_new, const int32_t* slot, int B, int n_kv,
                              int32_t* tail_len, int32_t* seq_len, int64_t S_cap, int64_t ovf_cap, int n_base_rows, int32_t* err, void* stream) {
  if (!K || !V || !k_new || !v_new || !slot || !tail_len || !seq_len) return GAAC_E_ARG;
  if (B <= 0 || n_kv <= 0 || S_cap <= 0 || S_cap % T || ovf_cap <= 0 || n_base_rows <= 0) return GAAC_E_ARG;
  for (const gaac_store* s : {K, V}) {
    if (!s->sm || !s->codes || !s->flags || !s->tile_off || !s->ovf || !s->ovf_used || !s->tail || !s->base3 || !s->base4) return GAAC_E_ARG;
    if (!aligned16(s->sm) || !aligned16(s->codes) || !aligned16(s->tail)) return GAAC_E_ALIGN;
  }
  if ((reinterpret_cast<uintptr_t>(k_new) & 7) || (reinterpret_cast<uintptr_t>(v_new) & 7)) return GAAC_E_ALIGN;
  AppendParams p{*K, *V, (const uint16_t*)k_new, (const uint16_t*)v_new, slot, n_kv, tail_len, seq_len, S_cap, ovf_cap, n_base_rows, err};
  return launch_overlapped(append_kv_kernel, dim3((unsigned)(B * n_kv)), 64, (cudaStream_t)stream, p);
}

extern "C" int gaac_paged_store(const gaac_paged* st, const void* key, const void* value, int64_t k_stride, int64_t v_stride,
                                const int32_t* ent, int E, int32_t* freeq, void* stream) {
  if (int e = check_paged(st)) return e;
  if (!key || !value || !ent || !freeq || E < 0 || k_stride < (int64_t)st->n_kv * D || v_stride < (int64_t)st->n_kv * D) return GAAC_E_ARG;
  if (!aligned16(key) || !aligned16(value) || k_stride % 8 || v_stride % 8) return GAAC_E_ALIGN;
  if (E == 0) return GAAC_OK;
  PagedParams p{*st, (const uint16_t*)key, (const uint16_t*)value, k_stride, v_stride, ent, freeq};
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t items = (int64_t)E * 2 * st->n_kv;
  if (items <= STEP_WARPS * STEP_CLUSTER) {
    unsigned blocks = 1;
    while (blocks * STEP_WARPS < items) blocks *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks); cfg.blockDim = dim3(STEP_WARPS * 32); cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = blocks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = g_launch_overlap;
    cfg.attrs = at; cfg.numAttrs = 2;
    if (cudaLaunchKernelEx(&cfg, paged_store_step_kernel, p, (int)items) != cudaSuccess) { cudaGetLastError(); return GAAC_E_LAUNCH; }
    return launch_status();
  }
  if (int err = launch_overlapped(paged_store_kernel, dim3((unsigned)E, (unsigned)(2 * st->n_kv)), 32, s, p)) return err;
  const int n = E * 2 * st->n_kv;
  return launch_overlapped(free_tiles_kernel, dim3((n + 255) / 256), 256, s, freeq, n, st->stack, st->top);
}

extern "C" int gaac_paged_release(const gaac_paged* st, const int32_t* blocks, int F, void* stream) {
  if (int e = check_paged(st)) return e;
  if (!blocks || F < 0) return GAAC_E_ARG;
  if (F == 0) return GAAC_OK;
  release_blocks_kernel<<<(unsigned)F, 32, 0, (cudaStream_t)stream>>>(blocks, 2 * st->n_kv, st->mt, st->stack, st->top);
  return launch_status();
}

extern "C" int gaac_paged_decode_blocks(const gaac_paged* st, const int32_t* pairs, int P, void* sk, void* sv, int64_t row_stride, void* stream) {
  if (int e = check_paged(st)) return e;
  if (!pairs || !sk || !sv || P < 0 || row_stride < (int64_t)st->n_kv * D) return GAAC_E_ARG;
  if (!aligned16(sk) || !aligned16(sv) || row_stride % 8) return GAAC_E_ALIGN;
  if (P == 0) return GAAC_OK;
  PagedDecodeParams p{*st, pairs, P, (uint16_t*)sk, (uint16_t*)sv, row_stride};
  return launch_overlapped_with(PDEC_WARPS * decode_scratch_bytes(std::min(st->ovf_slot, TILE_MAX_ESC)), PDEC_SHARED, paged_decode_blocks_kernel, dim3((unsigned)((P + PDEC_WARPS - 1) / PDEC_WARPS), (unsigned)(2 * st->n_kv)),
                                PDEC_WARPS * 32, (cudaStream_t)stream, p);
}

extern "C" const char* gaac_status_string(int status) {
  switch (status) {
    case GAAC_OK: return "ok";
    case GAAC_E_ARG: return "invalid argument (null pointer, bad size or inconsistent sizes)";
    case GAAC_E_UNSUPPORTED: return "unsupported configuration (GQA group must be 1..8, head_dim 128, tile stride a multiple of 16)";
    case GAAC_E_ALIGN: return "a buffer is not aligned as required";
    case GAAC_E_LAUNCH: return "CUDA launch failed";
    case GAAC_E_WORKSPACE: return "workspace missing or too small";
    default: return "unknown status";
  }
}

extern "C" int gaac_abi_version(void) { return GAAC_ABI_VERSION; }
