// Block encoder, escape-stream compaction, page decoder and calibration kernels (sm_100a).
#include <algorithm>
#include <atomic>
#include <mutex>
#include "gaac_api.cuh"
#include "gaac_warp.cuh"

namespace gaac {

constexpr int ENC_WARPS = 4;          // warps per CTA
// Tiles of a warp, which share the head's base words (and, in the decoder, the CTA's tables).  A launch that fits the SMs a few times over is as long as a warp's tiles take one after
// the other, so a warp has one while the CTAs are fewer than twice what the SMs hold, and more only as the waves of CTAs become many.
//  encoder (5 CTAs per SM)  us with 1 / 2 / 4 tiles: [8, 1111, 128] 3.3 / 4.2 / 6.3;  a prompt of 4001 tokens, 8 heads, K and V 8.0 / 8.2 / 9.2;  [8, 65536, 128] 47.4 / 42.3 / 41.7 (12: 46.1)
//  decoder (8 CTAs per SM)  [8, 4001, 128] 4.9 / 5.9 / 8.4;  [8, 65536, 128] K and V, two passes queued at once, 86.7 / 83.1 / 83.8 (7, every SM filled exactly once: 93.7)
constexpr int ENC_RESIDENT = 5 * 148, ENC_MOST = 4, DEC_RESIDENT = 8 * 148, DEC_MOST = 2;
static_assert(2 * DEC_MOST <= 32, "a lane for either end of each tile's escape bytes");
static int tiles_per_warp(int64_t ntiles, int64_t rows, int resident, int most) {
  const int64_t ctas = (ntiles + ENC_WARPS - 1) / ENC_WARPS * rows;
  return (int)std::max<int64_t>(1, std::min<int64_t>(most, ctas / resident));
}

// 2^40 escape bytes are those of 3.5 TB of BF16, 2^24 CTAs (of 16 tiles in a launch of so many, and at most one more per head) those of 1.1 TB: neither part overflows.
constexpr int DONE_SHIFT = 40;
constexpr int TOTAL_TOO_LARGE = -2;

// What one kind's encode reads and writes.
struct EncodeSide {
  const uint16_t* x; const uint8_t *base3, *base4;
  uint8_t *sm, *codes; int* flags; uint8_t* slots; int* tile_bytes;
  int* clear;                     // optional: a word that the first block sets to zero (the ticket of the scan, a status word)
  int* cta_bytes;                 // optional: escape bytes of the tiles of every CTA, [H][gridDim.x]
  unsigned long long* counter;    // optional: CTAs that are done << DONE_SHIFT | their escape bytes; zero on entry, left zero
  int* total;                     // with counter: the last CTA writes all escape bytes here (page-locked host memory), -2 for more than 31 bits hold
};
struct EncodeParams { EncodeSide side[2]; long S, x_head_stride, x_row_stride, S_pad; const int* bidx; int n_kv, ntiles, per_warp; };

// One warp per (head, tile).  Token t of head h is read at x + h * x_head_stride + t * x_row_stride (bf16 elements): head-major [H, S_in, 128] or
// token-major [L, n_kv, 128] input.
template <int KIND_V>
__device__ __forceinline__ void encode_tiles_cta(const EncodeParams& p, const EncodeSide& s, WarpScratch (*scratch)[ENC_WARPS], uint8_t* esc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ntiles = p.ntiles;
  const long h = blockIdx.y;
  if (s.clear && blockIdx.x == 0 && h == 0 && threadIdx.x == 0) *s.clear = 0;
  const int brow = p.bidx ? p.bidx[h] : (int)(h % p.n_kv);
  u32 b3w[8], b4w[8];
  load_base_words<KIND_V>(s.base3 + (long)brow * D, s.base4 + (long)brow * D, lane, b3w, b4w);
  const int tile0 = blockIdx.x * (ENC_WARPS * p.per_warp) + warp;
  const uint16_t* xh = s.x + h * p.x_head_stride;
  auto fetch = [&](int i) {                           // rows of the warp's i-th tile into scratch[i & 1]
    const long row0 = (long)(tile0 + i * ENC_WARPS) * T;
    stage_rows_async(scratch[i & 1][warp], xh + row0 * p.x_row_stride, p.x_row_stride, (int)min((long)T, p.S - row0), lane);
    async_commit();
  };
  if (tile0 < ntiles) fetch(0);
  int sum = 0;
  for (int i = 0; i < p.per_warp; i++) {
    const int tile = tile0 + i * ENC_WARPS;
    if (tile >= ntiles) break;                       // warp-uniform
    const bool more = i + 1 < p.per_warp && tile + ENC_WARPS < ntiles;
    __syncwarp();                                    // the other scratch was read by the tile before this one
    if (more) { fetch(i + 1); async_wait<1>(); } else async_wait<0>();
    WarpScratch& ws = scratch[i & 1][warp];
    const long row0 = (long)tile * T;
    const int nvalid = (int)min((long)T, p.S - row0);
    LaneTile lt;
    const int total = encode_tile_warp<KIND_V>(ws, nvalid, b3w, b4w, lane, lt);
    const long trow = h * p.S_pad + row0;
    store_tile_payload<KIND_V>(lt, s.sm + trow * D, s.codes + trow * CB, reinterpret_cast<uint8_t*>(s.flags + trow), lane);
    // escape bytes: gathered in shared memory with byte stores (every lane at its own positions), then written to the tile's
    // scratch slot as whole words by neighbouring lanes, so the slot costs one or two coalesced stores instead of ~50 byte stores
    store_tile_escapes<KIND_V>(ws, lt, esc, lane);
    __syncwarp();
    {
      u32* dst = reinterpret_cast<u32*>(s.slots + (h * ntiles + tile) * (long)TILE_MAX_ESC);
      const u32* src = reinterpret_cast<const u32*>(esc);
      for (int k = lane; 4 * k < total; k += 32) dst[k] = src[k];
    }
    if (lane == 0) s.tile_bytes[h * ntiles + tile] = total;
    sum += total;
  }
  if (s.cta_bytes || s.counter) {
    __shared__ int warp_sum[ENC_WARPS];
    if (lane == 0) warp_sum[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      int all = 0;
#pragma unroll
      for (int w = 0; w < ENC_WARPS; w++) all += warp_sum[w];
      if (s.cta_bytes) s.cta_bytes[h * gridDim.x + blockIdx.x] = all;
      if (s.counter) {
        const unsigned long long before = atomicAdd(s.counter, 1ull << DONE_SHIFT | (u32)all);
        if ((u32)(before >> DONE_SHIFT) == gridDim.x * gridDim.y - 1u) {
          const unsigned long long bytes = (before & ((1ull << DONE_SHIFT) - 1)) + (u32)all;
          *s.counter = 0ull;
          *(volatile int*)s.total = bytes > 0x7FFFFFFFull ? TOTAL_TOO_LARGE : (int)bytes;
        }
      }
    }
  }
}
// KIND 0 / 1: K or V alone, grid = (ceil(ntiles / (4 * per_warp)), H).  2: both, grid z = kind (a prompt's K and V: one launch, and short prompts leave
// half as much of the GPU idle).
template <int KIND>
__global__ void __launch_bounds__(ENC_WARPS * 32) encode_tiles_kernel(const __grid_constant__ EncodeParams p) {
  __shared__ __align__(16) WarpScratch scratch[2][ENC_WARPS];       // two per warp: the next tile's rows arrive while this one is encoded
  __shared__ __align__(16) uint8_t esc_stage[ENC_WARPS][TILE_MAX_ESC];
  griddep_wait();
  griddep_launch();
  const bool v = KIND == 2 ? blockIdx.z != 0 : KIND == 1;
  if (KIND != 0 && v) encode_tiles_cta<1>(p, p.side[KIND == 2 ? 1 : 0], scratch, esc_stage[threadIdx.x >> 5]);
  if (KIND != 1 && !v) encode_tiles_cta<0>(p, p.side[0], scratch, esc_stage[threadIdx.x >> 5]);
}
static dim3 encode_grid(int ntiles, int64_t H, int kinds, int per_warp) { return dim3((ntiles + ENC_WARPS * per_warp - 1) / (ENC_WARPS * per_warp), (unsigned)H, (unsigned)kinds); }

// head_start[0..H] = exclusive prefix of head_bytes, by one CTA of SCAN_THREADS threads (H is the number of cache heads).
// total: optional, the sum once more (page-locked host memory, which the end of the kernel makes visible).
__device__ __forceinline__ void head_prefix(const int* head_bytes, int H, int* head_start, int* total) {
  __shared__ int hsum[32];
  __shared__ int hcarry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (H <= 64) {                                     // the usual case: one warp, no barriers
    if (warp) return;
    int carry = 0;
    for (int base = 0; base < H; base += 32) {
      int inc = base + lane < H ? __ldcg(head_bytes + base + lane) : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) { int u = __shfl_up_sync(FULL, inc, d); if (lane >= d) inc += u; }
      if (base + lane < H) head_start[base + lane + 1] = carry + inc;
      carry += __shfl_sync(FULL, inc, 31);
    }
    if (lane == 0) head_start[0] = 0;
    if (total && lane == 0) *(volatile int*)total = carry;
    return;
  }
  if (tid == 0) { hcarry = 0; head_start[0] = 0; }
  __syncthreads();
  for (int base = 0; base < H; base += blockDim.x) {
    const int i = base + tid;
    int inc = i < H ? __ldcg(head_bytes + i) : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { int u = __shfl_up_sync(FULL, inc, d); if (lane >= d) inc += u; }
    if (lane == 31) hsum[warp] = inc;
    __syncthreads();
    int before = hcarry;
    for (int w = 0; w < warp; w++) before += hsum[w];
    if (i < H) head_start[i + 1] = before + inc;
    __syncthreads();
    if (tid == (int)blockDim.x - 1) hcarry = before + inc;
    __syncthreads();
  }
  if (total && tid == 0) *(volatile int*)total = hcarry;
}

// Exclusive prefix of tile_bytes per head.  One CTA of 1024 threads per (head, kind), four tiles per thread and pass: a 64K-token
// head (4096 tiles) is one pass of two warp scans.  With head_start (one kind) the CTA that finishes last also makes the prefix over the
// heads, head_start[0..H], and hands head_start[H] to the host through `total` (pinned memory, may be NULL): a launch and a copy less than
// doing it behind this kernel.  head_start[H] is the ticket until then and must be zero on entry.
struct ScanSide { const int* tile_bytes; int *tile_off, *head_bytes; };
struct ScanParams { ScanSide side[2]; int ntiles; long tile_off_stride; int* head_start; int* total; };
constexpr int SCAN_THREADS = 1024;
__global__ void __launch_bounds__(SCAN_THREADS) tile_scan_kernel(const __grid_constant__ ScanParams p) {
  const int* tile_bytes = p.side[blockIdx.y].tile_bytes;
  int* tile_off = p.side[blockIdx.y].tile_off;
  int* head_bytes = p.side[blockIdx.y].head_bytes;
  const int ntiles = p.ntiles;
  const long tile_off_stride = p.tile_off_stride;
  __shared__ int wsum[32];
  __shared__ int carry_s, pass_total;
  const long h = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry_s = 0;
  griddep_wait();
  griddep_launch();
  __syncthreads();
  for (int base = 0; base < ntiles; base += 4 * SCAN_THREADS) {
    const int i0 = base + 4 * tid;
    int v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = i0 + k < ntiles ? tile_bytes[h * ntiles + i0 + k] : 0;
    const int s = v[0] + v[1] + v[2] + v[3];
    int inc = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { int u = __shfl_up_sync(FULL, inc, d); if (lane >= d) inc += u; }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      const int w = wsum[lane];
      int winc = w;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) { int u = __shfl_up_sync(FULL, winc, d); if (lane >= d) winc += u; }
      wsum[lane] = winc - w;                         // exclusive prefix over the warps
      if (lane == 31) pass_total = winc;
    }
    __syncthreads();
    int off = carry_s + wsum[warp] + inc - s;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (i0 + k < ntiles) tile_off[h * tile_off_stride + i0 + k] = off;
      off += v[k];
    }
    __syncthreads();
    if (tid == 0) carry_s += pass_total;
    __syncthreads();
  }
  if (tid == 0 && head_bytes) head_bytes[h] = carry_s;
  if (!p.head_start) return;
  __shared__ int last;
  const int H = gridDim.x;
  if (tid == 0) { __threadfence(); last = atomicAdd(p.head_start + H, 1) == H - 1; }
  __syncthreads();
  if (!last) return;
  __threadfence();
  head_prefix(head_bytes, H, p.head_start, p.total);
}

__global__ void __launch_bounds__(SCAN_THREADS) head_prefix_kernel(const int* __restrict__ head_bytes, int H, int* __restrict__ head_start) { head_prefix(head_bytes, H, head_start, nullptr); }

// What one kind's compaction reads and writes.
struct CompactSide { const uint8_t* slots; const int *tile_bytes, *tile_off, *head_start; uint8_t* ovf; const int* flags; int* ovf_off; int* status; };
struct CompactParams { CompactSide side[2]; int ntiles; unsigned n_items; long tile_off_stride, head_stride, S, S_pad; int zero_pad; long ovf_cap, head_cap; };

// Escape bytes of every tile: slot -> ovf[head_start[h] + tile_off[h, tile]]; optionally the per-row escape offsets
// ovf_off[h, row] = tile_off[h, tile] + (escape bytes of the tile's earlier rows), recomputed from the tag words.
// Eight lanes per tile: a tile has some 55 escape bytes and 16 tag words, and what the kernel waits for are its loads (sizes and offsets, then the
// bytes), so a warp keeps four tiles in flight.  grid y = kind.
__global__ void __launch_bounds__(128) compact_copy_kernel(const __grid_constant__ CompactParams p) {
  griddep_wait();
  const CompactSide& s = p.side[blockIdx.y];
  const int lane = threadIdx.x & 31, q = lane & 7;
  const unsigned first = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 4, item = first + (lane >> 3);
  const bool live = item < p.n_items;
  const unsigned h = live ? item / (unsigned)p.ntiles : 0u, t = live ? item - h * (unsigned)p.ntiles : 0u;
  const int n = live ? s.tile_bytes[item] : 0;
  const int toff = live ? s.tile_off[h * p.tile_off_stride + t] : 0;
  const uint8_t* src = s.slots + (long)item * TILE_MAX_ESC;
  // bounds: the whole stream must fit ovf_cap bytes (ovf_cap > 0), a head's part head_cap bytes (head_cap > 0), read padding
  // included; a tile that does not fit is not written and bit 0 of *status is set.  Offsets below zero are those of a stream that 31 bits cannot count: they fit nowhere.
  const long at = (s.head_start ? (long)s.head_start[h] : (long)h * p.head_stride) + toff;        // no table: head h's stream starts at h * head_stride
  const bool fits = at >= 0 && toff >= 0 && (p.ovf_cap <= 0 || at + n + p.zero_pad <= p.ovf_cap) && (p.head_cap <= 0 || (long)toff + n + p.zero_pad <= p.head_cap);
  if (fits) {
    uint8_t* dst = s.ovf + at;
#pragma unroll 4
    for (int i = q; i < n; i += 8) dst[i] = src[i];
  } else if (live && q == 0 && s.status) atomicOr(s.status, 1);
  if (p.zero_pad && p.head_cap <= 0 && s.head_start && first == 0 && lane < p.zero_pad) {                              // over-read padding behind the last head (packed stream)
    const long end = (long)s.head_start[p.n_items / (unsigned)p.ntiles];
    if (end >= 0 && (p.ovf_cap <= 0 || end + p.zero_pad <= p.ovf_cap)) s.ovf[end + lane] = 0;
    else if (lane == 0 && s.status) atomicOr(s.status, 1);
  }
  if (s.ovf_off) {
    const long row = (long)t * T + 2 * q;
    const int s0 = live && row < p.S ? row_esc_bytes((u32)s.flags[h * p.S_pad + row]) : 0, s1 = live && row + 1 < p.S ? row_esc_bytes((u32)s.flags[h * p.S_pad + row + 1]) : 0;
    int inc = s0 + s1;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) { const int v = __shfl_up_sync(FULL, inc, d, 8); if (q >= d) inc += v; }
    int* o = s.ovf_off + (long)h * p.S + row;
    if (live && row < p.S) o[0] = toff + inc - s0 - s1;
    if (live && row + 1 < p.S) o[1] = toff + inc - s1;
  }
}
static dim3 compact_grid(const CompactParams& p, int kinds) { return dim3((p.n_items + 15) / 16, (unsigned)kinds); }

// One warp per (head, tile): compressed tile -> bf16 rows.  Bound by latency and the warps that hide it: the escape bytes are asked for with the tile, their number taken from
// the offset of the next tile (not of a head's last one), and the registers leave room for 8 CTAs of K, 7 of V.  [8, 65536, 128] K and V: 98.5 -> 93.7 us; with 6
// CTAs each 102, and with the next tile's words asked for while one is rebuilt (5 CTAs) 101.  Launched overlapped, with two tiles per warp: 90.3 -> 83.1 for two
// passes over K and V queued at once (the public calls, over three Pages in turn: 90.6 -> 88.7).  No help: 32-byte
// stores (85.6), evict-first stores (83.5) or loads (85.4), CTAs of two warps (92.6).
template <int KIND_V>
__global__ void __launch_bounds__(ENC_WARPS * 32, KIND_V ? 7 : 8) decode_page_kernel(
    const uint8_t* __restrict__ sm, const uint8_t* __restrict__ codes, const int* __restrict__ flags, const int* __restrict__ tile_off,
    long tile_off_stride, const uint8_t* __restrict__ ovf, const int* __restrict__ head_start, const uint8_t* __restrict__ base3,
    const uint8_t* __restrict__ base4, const int* __restrict__ bidx, int n_kv, long S, long S_pad, uint16_t* __restrict__ out, int ntiles, int per_warp) {
  __shared__ __align__(16) uint8_t scratch[ENC_WARPS * decode_scratch_bytes(TILE_MAX_ESC)];
  __shared__ __align__(16) DecodeTables tables;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long h = blockIdx.y;
  WarpScratch& ws = *reinterpret_cast<WarpScratch*>(scratch + warp * decode_scratch_bytes(TILE_MAX_ESC));
  griddep_wait();
  griddep_launch();
  const int brow = bidx ? bidx[h] : h < n_kv ? (int)h : (int)((unsigned)h % (unsigned)n_kv);
  const uint8_t* esc_head = ovf + (long)head_start[h];
  const int tile0 = blockIdx.x * (ENC_WARPS * per_warp) + warp;
  const int mine = tile0 + (lane >> 1) * ENC_WARPS + (lane & 1);                           // lanes 2i, 2i + 1: where the warp's i-th tile's escape bytes begin and end
  const int off = lane < 2 * per_warp && mine < ntiles ? tile_off[h * tile_off_stride + mine] : 0;
  TileWords<KIND_V> tw;
  const auto ask = [&](int i) {                       // the words of the warp's i-th tile, escape bytes included where the next tile's offset says how many
    const int tile = tile0 + i * ENC_WARPS, from = __shfl_sync(FULL, off, 2 * i), to = __shfl_sync(FULL, off, 2 * i + 1);
    const long trow = h * S_pad + (long)tile * T;
    load_tile_words<KIND_V>(tw, sm + trow * D, codes + trow * CB, reinterpret_cast<const uint8_t*>(flags + trow), esc_head + from, tile + 1 < ntiles ? to - from : 0, lane);
  };
  if (tile0 < ntiles) ask(0);
  const u32 w = fill_decode_tables<KIND_V>(tables, base3 + (long)brow * D, base4 + (long)brow * D);
  __syncthreads();
#pragma unroll 1
  for (int i = 0; i < per_warp; i++) {
    const int tile = tile0 + i * ENC_WARPS;
    if (tile >= ntiles) break;
    const long row0 = (long)tile * T;
    if (i) ask(i);
    decode_tile_warp<KIND_V>(ws, tw, w, lane);
    unstage_rows(ws, out + (h * S + row0) * D, D, (int)min((long)T, S - row0), lane);
  }
}

// Exponent histogram: x [N rows, n_ch] bf16, row r at x + r * row_stride; counts of channel c at hist + c * PER_CHANNEL.  grid = (ceil(n_ch/128), row chunks, kinds).  A CTA
// counts 128 channels in shared memory with 8-bit counters and flushes what is not zero with atomics.  Counter (bin, place) is byte bin & 3 of word
// [bin >> 2][place]: a warp's increments go to 32 banks whatever the exponents are, and clearing and flushing handle four bins at a time, nearly all of them empty.  PAIRS
// (even strides, rows on 4-byte boundaries): a thread reads two neighbouring channels with one load, whose places are 64 apart.
// Bound by latency and by the atomics of the flush, which go to a line each: so the prompt's histogram has 16-bit counts, four to a 64-bit atomic (Packed: prompts of up to 65535
// tokens), which is a third of the atomics.  With one thread per channel and a load, add and store per value it took 21 us for 2048 rows of 8 kv heads (15 us with
// 16-bit counters and chunks of 64 rows), 7 us as shared-memory atomics that return nothing.
// Rows per CTA (an 8-bit counter holds 255) and threads.  us of a prompt's tables, 8 heads x 4001 tokens / 8 x 32768 / 1 x 4096: 128 rows, 256 threads 11.7 / 44 / 6.7;  512 threads 13.0 / 46 /
// 6.2;  192 rows 11.8 / 41 / 7.2;  96 rows 12.7 / 49 / 6.5;  before, one channel per load and 32-bit counts 15.2 / 65 / 7.6.
constexpr int HIST_ROWS = 128, HIST_THREADS = 256;
typedef unsigned long long u64_t;
struct Packed { u64_t four; };                        // counts of bins 4w .. 4w + 3, 16 bits each
template <class Cnt> constexpr int PER_CHANNEL = 256;
template <> constexpr int PER_CHANNEL<Packed> = 64;
template <class Cnt> struct HistParams { const uint16_t* x[2]; Cnt* hist[2]; long N, n_ch, row_stride; };
__device__ __forceinline__ void add_four(Packed* hist, int w, u32 four) { atomicAdd(&hist[w].four, (u64_t)prmt(four, 0u, 0x4140) | (u64_t)prmt(four, 0u, 0x4342) << 32); }
template <class Cnt> __device__ __forceinline__ void add_four(Cnt* hist, int w, u32 four) {
#pragma unroll
  for (int i = 0; i < 4; i++) { const u32 n = (four >> (8 * i)) & 0xFFu; if (n) atomicAdd(&hist[4 * w + i], (Cnt)n); }
}
// A thread's rows of the CTA's chunk: x is at its channels' first value, col, sub its place in the CTA.
template <bool PAIRS> __device__ __forceinline__ void count_rows(u32 (&bins)[64][128], const uint16_t* x, long N, long row_stride, int col, int sub) {
  constexpr int LANES = HIST_THREADS / (PAIRS ? 64 : 128);
  const auto load = [&](long r) -> u32 { return PAIRS ? *reinterpret_cast<const u32*>(x + r * row_stride) : x[r * row_stride]; };
  const auto count = [&](u32 v) {                     // exponent = bits 7..14
    atomicAdd(&bins[(v >> 9) & 0x3Fu][col], 1u << (8u * ((v >> 7) & 3u)));
    if (PAIRS) atomicAdd(&bins[(v >> 25) & 0x3Fu][64 + col], 1u << (8u * ((v >> 23) & 3u)));
  };
  const long r1 = min(N, ((long)blockIdx.y + 1) * HIST_ROWS);
  long r = (long)blockIdx.y * HIST_ROWS + sub;
  for (; r + 15 * LANES < r1; r += 16 * LANES) {      // sixteen independent loads in flight per thread
    u32 v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = load(r + i * LANES);
#pragma unroll
    for (int i = 0; i < 16; i++) count(v[i]);
  }
  for (; r < r1; r += LANES) count(load(r));
}
// Behind clear_kernel x was there before that kernel, so the counting need not wait for it, only the flush (EARLY).
template <class Cnt, bool PAIRS, bool EARLY>
__global__ void __launch_bounds__(HIST_THREADS) exponent_hist_kernel(const __grid_constant__ HistParams<Cnt> p) {
  __shared__ __align__(16) u32 bins[64][128];
  constexpr int WIDE = PAIRS ? 2 : 1, COLS = 128 / WIDE;                                   // channels of a thread, threads side by side
  const int col = threadIdx.x % COLS, sub = threadIdx.x / COLS;
  const long c = (long)blockIdx.x * 128 + WIDE * col;
  for (int i = threadIdx.x; i < 64 * 128 / 4; i += HIST_THREADS) reinterpret_cast<uint4*>(bins)[i] = make_uint4(0, 0, 0, 0);
  if (!EARLY) griddep_wait();
  griddep_launch();
  __syncthreads();
  if (c < p.n_ch) count_rows<PAIRS>(bins, p.x[blockIdx.z] + c, p.N, p.row_stride, col, sub);
  __syncthreads();
  const int place = threadIdx.x & 127;
  const long ch = (long)blockIdx.x * 128 + (PAIRS ? 2 * (place & 63) + (place >> 6) : place);
  if (EARLY) griddep_wait();
  if (ch >= p.n_ch) return;
  Cnt* hist = p.hist[blockIdx.z] + ch * PER_CHANNEL<Cnt>;
#pragma unroll 8
  for (int w = threadIdx.x >> 7; w < 64; w += HIST_THREADS / 128) {
    const u32 four = bins[w][place];
    if (four) add_four(hist, w, four);
  }
}
// The counters of a prompt's histogram cleared (a kernel and not a memset, so that the counting need not wait for it).
__global__ void __launch_bounds__(256) clear_kernel(u32* p, int n) {
  griddep_launch();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) p[i] = 0u;
}

// One warp per histogram row: densest 8- and 16-wide window, first maximum wins.  grid y = kind.  A lane has eight neighbouring bins, so one scan over the lanes makes the prefix.
template <class Cnt> struct BasesParams { const Cnt* hist[2]; uint8_t *base3[2], *base4[2]; long n_rows; bool clear; };       // clear: the counters are left zero
template <class Cnt> struct Counts {
  typedef Cnt Sum;
  static __device__ __forceinline__ void load(const Cnt* row, int lane, Cnt (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = row[8 * lane + i];
  }
  static __device__ __forceinline__ void clear(Cnt*, int) {}
};
template <> struct Counts<Packed> {
  typedef int Sum;
  static __device__ __forceinline__ void load(const Packed* row, int lane, int (&v)[8]) {
    const uint4 q = reinterpret_cast<const uint4*>(row)[lane];
    const u32 w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = (int)((w[i >> 1] >> (16 * (i & 1))) & 0xFFFFu);
  }
  static __device__ __forceinline__ void clear(Packed* row, int lane) { reinterpret_cast<uint4*>(row)[lane] = make_uint4(0u, 0u, 0u, 0u); }
};
template <class Cnt>
__global__ void __launch_bounds__(128) bases_from_hist_kernel(const __grid_constant__ BasesParams<Cnt> p) {
  typedef typename Counts<Cnt>::Sum Sum;
  __shared__ Sum cs[4][256 + 8 + 1];                  // [row of the CTA][bin + (bin >> 5)]: prefix of the counts, the lanes' eights in different banks
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * 4 + warp;
  griddep_wait();
  griddep_launch();
  if (row >= p.n_rows) return;
  Sum v[8], own = 0;
  Counts<Cnt>::load(p.hist[blockIdx.y] + row * PER_CHANNEL<Cnt>, lane, v);
  if (p.clear) Counts<Cnt>::clear(const_cast<Cnt*>(p.hist[blockIdx.y]) + row * PER_CHANNEL<Cnt>, lane);
#pragma unroll
  for (int i = 0; i < 8; i++) own += v[i];
  Sum inc = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) { const Sum u = __shfl_up_sync(FULL, inc, d); if (lane >= d) inc += u; }
  const auto at = [](int bin) { return bin + (bin >> 5); };
  Sum before = inc - own;
#pragma unroll
  for (int i = 0; i < 8; i++) { cs[warp][at(8 * lane + i)] = before; before += v[i]; }
  if (lane == 31) cs[warp][at(256)] = before;
  __syncwarp();
  for (int k = 0; k < 2; k++) {
    const int w = k ? 16 : 8;
    Sum best = -1; int besti = 0;
    for (int s = lane; s <= 256 - w; s += 32) {
      const Sum n = cs[warp][at(s + w)] - cs[warp][at(s)];
      if (n > best) { best = n; besti = s; }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const Sum ob = __shfl_xor_sync(FULL, best, d); const int oi = __shfl_xor_sync(FULL, besti, d);
      if (ob > best || (ob == best && oi < besti)) { best = ob; besti = oi; }
    }
    if (lane == 0) (k ? p.base4[blockIdx.y] : p.base3[blockIdx.y])[row] = (uint8_t)besti;
  }
}

// ---- end of a slot's prefill: offsets, escape bytes, tails and counters in ONE launch behind the encode.
struct FinishSide { const uint8_t* slots; const int *tile_bytes, *cta_bytes; int* tile_off; uint8_t* ovf; int *used, *status; const uint16_t* tok; uint16_t* tail; };       // (used, ovf, ..: of the slot's heads)
struct FinishParams { FinishSide side[2]; long L, row_stride, tile_off_stride, ovf_cap, head_cap; int n_kv, ntiles, per_cta, ctas, chunk, chunks; int *seq_len, *tail_len; };
constexpr int FINISH_THREADS = 128, FINISH_TILES = FINISH_THREADS / 8, FINISH_STAGE = 128 * FINISH_TILES;

// The prompt's remainder (L mod 16 rows) goes into the head's raw tail, the head's counters are set; the block of head 0 also has the heads' escape bytes from the encoder's
// sums and reports the largest for the host's capacity check.
__device__ __forceinline__ void finish_head(const FinishParams& p, const FinishSide& s, int h, int kind) {
  const long n_full = p.L / T * T;
  const int rem = (int)(p.L - n_full), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint16_t* src = s.tok + n_full * p.row_stride + h * D;
  uint16_t* dst = s.tail + (long)h * T * D;
#pragma unroll
  for (int i = tid; i < T * 16; i += FINISH_THREADS)
    if ((i >> 4) < rem) *reinterpret_cast<uint4*>(dst + i * 8) = *reinterpret_cast<const uint4*>(src + (i >> 4) * p.row_stride + (i & 15) * 8);
  if (tid == 0 && kind == 0) { p.seq_len[h] = (int)n_full; p.tail_len[h] = rem; }
  if (h) return;
  __shared__ int most[FINISH_THREADS / 32];
  int m = 0;
  for (int k = warp; k < p.n_kv; k += FINISH_THREADS / 32) {
    int n = 0;
    for (int i = lane; i < p.ctas; i += 32) n += s.cta_bytes[(long)k * p.ctas + i];
    n = __reduce_add_sync(FULL, n);
    if (lane == 0) s.used[k] = n;
    m = max(m, n);
  }
  if (lane == 0) most[warp] = m;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < FINISH_THREADS / 32; w++) m = max(m, most[w]);
    s.status[1] = m;
    if (p.ntiles == 0) s.status[0] = 0;              // (no encode in front that cleared it)
  }
}
// A block has `chunk` tiles of a head (up to 16, whole CTAs of the encoder), eight lanes per tile.  Where they begin in the head's stream is the sum of what the encoder's CTAs before them have, where
// a tile begins follows from a scan over the block, and the bytes go through shared memory so that they leave in 16-byte stores.  Bound by latency, so everything that is
// read is asked for at once, the first 64 bytes of a tile's slot (55 is usual) before their number is known, and blocks are small: 4001 tokens of 8 heads
// with 64 tiles each 3.7 us, now 3.4;  the whole prompt with every group raw 39, now 28.  A prompt of 8 heads with its tables in four launches (encode, this, histogram, windows) against six (a clear, and
// offsets and copy apart): 500 tokens 19.8 -> 12.7 us, 4001 30.9 -> 22.4, 32768 113 -> 87;  every group raw 25 -> 14, 31 -> 28, 90 -> 90 (without tables).
__global__ void __launch_bounds__(FINISH_THREADS) prefill_finish_kernel(const __grid_constant__ FinishParams p) {
  __shared__ __align__(16) uint8_t stage[FINISH_STAGE + 16];
  __shared__ int warp_tiles[FINISH_THREADS / 32], warp_before[FINISH_THREADS / 32];
  const FinishSide& s = p.side[blockIdx.y];
  griddep_wait();
  griddep_launch();
  const int copies = p.n_kv * p.chunks;
  if ((int)blockIdx.x >= copies) { finish_head(p, s, blockIdx.x - copies, blockIdx.y); return; }
  const int h = blockIdx.x / p.chunks, tile0 = (blockIdx.x % p.chunks) * p.chunk, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = tid >> 3, q = tid & 7;
  const bool live = t < min(p.chunk, p.ntiles - tile0);
  const long item = (long)h * p.ntiles + tile0 + t;
  const uint8_t* slot = s.slots + item * TILE_MAX_ESC;
  const int n = live ? s.tile_bytes[item] : 0;
  u32 first[2] = {0u, 0u};
  if (live) { first[0] = reinterpret_cast<const u32*>(slot)[2 * q]; first[1] = reinterpret_cast<const u32*>(slot)[2 * q + 1]; }
  int part = 0;
  for (int i = tid; i < tile0 / p.per_cta; i += FINISH_THREADS) part += s.cta_bytes[(long)h * p.ctas + i];
  int inc = n;                                       // of the warp's tiles up to this one
#pragma unroll
  for (int d = 8; d < 32; d <<= 1) { const int v = __shfl_up_sync(FULL, inc, d); if (lane >= d) inc += v; }
  part = __reduce_add_sync(FULL, part);
  if (lane == 31) { warp_tiles[warp] = inc; warp_before[warp] = part; }
  __syncthreads();
  int begin = 0, local = inc - n, total = 0;         // of the block inside the head, of the tile inside the block
#pragma unroll
  for (int w = 0; w < FINISH_THREADS / 32; w++) { begin += warp_before[w]; if (w < warp) local += warp_tiles[w]; total += warp_tiles[w]; }
  if (live && q == 0) s.tile_off[h * p.tile_off_stride + tile0 + t] = begin + local;
  uint8_t* const dst = s.ovf + (long)h * p.ovf_cap + begin;
  if (total > FINISH_STAGE || (long)begin + total > p.head_cap) {           // more than the stage holds, or some tiles do not fit the head's share: these are not written
    const bool fits = (long)begin + local + n <= p.head_cap;
    if (!fits && live && q == 0) atomicOr(s.status, 1);
    for (int k = 0; k < 4; k++) {                    // the warp's tiles one by one: words of the destination out of two of the slot
      const int size = __shfl_sync(FULL, fits ? n : 0, 8 * k);
      uint8_t* const d = dst + __shfl_sync(FULL, local, 8 * k);
      const uint8_t* const b = s.slots + (item - t + 4 * warp + k) * TILE_MAX_ESC;
      const int odd = min(size, (int)(-reinterpret_cast<uintptr_t>(d) & 3)), words = (size - odd) >> 2, rest = odd + 4 * words;
      const u32* const from = reinterpret_cast<const u32*>(b);
      for (int i = lane; i < words; i += 32 * 5) {     // (five loads that do not wait for the stores)
        u32 v[5];
#pragma unroll
        for (int j = 0; j < 5; j++)
          if (i + 32 * j < words) v[j] = odd ? __funnelshift_r(from[i + 32 * j], from[i + 32 * j + 1], 8 * odd) : from[i + 32 * j];
#pragma unroll
        for (int j = 0; j < 5; j++)
          if (i + 32 * j < words) reinterpret_cast<u32*>(d + odd)[i + 32 * j] = v[j];
      }
      if (lane < odd) d[lane] = b[lane];
      if (rest + lane < size) d[rest + lane] = b[rest + lane];
    }
    return;
  }
  const int phase = (int)(reinterpret_cast<uintptr_t>(dst) & 15);
  uint8_t* const to = stage + phase + local;
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (8 * q + i < n) to[8 * q + i] = (uint8_t)(first[i >> 2] >> (8 * (i & 3)));
  for (int i = 64 + q; i < n; i += 8) to[i] = slot[i];
  __syncthreads();
  for (int k = tid; 16 * k < phase + total; k += FINISH_THREADS) {
    uint8_t* const line = dst - phase + 16 * k;
    if (16 * k >= phase && 16 * k + 16 <= phase + total) *reinterpret_cast<uint4*>(line) = reinterpret_cast<const uint4*>(stage)[k];
    else for (int i = max(0, phase - 16 * k); i < min(16, phase + total - 16 * k); i++) line[i] = stage[16 * k + i];
  }
}

}  // namespace gaac

using namespace gaac;

// gaac_encode_tiles with a word that the kernel clears
static int encode_tiles(const void* x_bf16, int64_t H, int64_t S, int64_t S_in, int64_t S_pad, const uint8_t* base3, const uint8_t* base4, const int32_t* bidx, int n_kv, int kind,
                        uint8_t* sm, uint8_t* codes, int32_t* flags, uint8_t* slots, int32_t* tile_bytes, int32_t* clear, void* stream,
                        unsigned long long* counter = nullptr, int32_t* total = nullptr) {
  if (!x_bf16 || !base3 || !base4 || !sm || !codes || !flags || !slots || !tile_bytes) return GAAC_E_ARG;
  if (H <= 0 || S <= 0 || S_in < S || S_pad < (S + T - 1) / T * T || S_pad % T || n_kv <= 0 || H > 65535 || (kind != GAAC_KIND_K && kind != GAAC_KIND_V)) return GAAC_E_ARG;
  if (!aligned16(x_bf16) || !aligned16(sm) || !aligned16(codes)) return GAAC_E_ALIGN;
  const int ntiles = (int)((S + T - 1) / T);
  const EncodeParams p{{{(const uint16_t*)x_bf16, base3, base4, sm, codes, flags, slots, tile_bytes, clear, nullptr, counter, total}, {}}, S, S_in * D, D, S_pad, bidx, n_kv, ntiles, tiles_per_warp(ntiles, H, ENC_RESIDENT, ENC_MOST)};
  return launch_overlapped(kind == GAAC_KIND_K ? encode_tiles_kernel<0> : encode_tiles_kernel<1>, encode_grid(ntiles, H, 1, p.per_warp), ENC_WARPS * 32, (cudaStream_t)stream, p);
}

extern "C" int gaac_encode_tiles(const void* x_bf16, int64_t H, int64_t S, int64_t S_in, int64_t S_pad,
                                 const uint8_t* base3, const uint8_t* base4, const int32_t* bidx, int n_kv, int kind,
                                 uint8_t* sm, uint8_t* codes, int32_t* flags, uint8_t* slots, int32_t* tile_bytes, void* stream) {
  return encode_tiles(x_bf16, H, S, S_in, S_pad, base3, base4, bidx, n_kv, kind, sm, codes, flags, slots, tile_bytes, nullptr, stream);
}

extern "C" int gaac_compact(const uint8_t* slots, const int32_t* tile_bytes, int64_t H, int64_t ntiles, const int32_t* head_start,
                            uint8_t* ovf, int32_t* tile_off, int64_t tile_off_stride, int32_t* head_bytes,
                            const int32_t* flags, int64_t S, int64_t S_pad, int32_t* ovf_off, void* stream) {
  if (!tile_bytes || !tile_off || H <= 0 || ntiles <= 0 || tile_off_stride < ntiles) return GAAC_E_ARG;
  if (head_start && (!ovf || !slots)) return GAAC_E_ARG;
  if (ovf_off && (!head_start || !flags || S <= 0 || S_pad < S)) return GAAC_E_ARG;
  if (int e = launch_overlapped(tile_scan_kernel, dim3((unsigned)H), SCAN_THREADS, (cudaStream_t)stream, ScanParams{{{tile_bytes, tile_off, head_bytes}, {}}, (int)ntiles, tile_off_stride, nullptr, nullptr})) return e;
  if (head_start) return gaac_compact_copy(slots, tile_bytes, H, ntiles, head_start, ovf, tile_off, tile_off_stride, flags, S, S_pad, ovf_off, 0, 0, 0, nullptr, stream);
  return launch_status();
}

static int encode_begin(const void* x_bf16, int64_t H, int64_t S, int64_t S_in, int64_t S_pad, const uint8_t* base3, const uint8_t* base4, const int32_t* bidx, int n_kv, int kind,
                        uint8_t* sm, uint8_t* codes, int32_t* flags, uint8_t* slots, int32_t* tile_bytes, int32_t* tile_off, int32_t* head_bytes, int32_t* head_start,
                        int32_t* total, void* stream) {
  if (!tile_off || !head_bytes || !head_start) return GAAC_E_ARG;
  if (int e = encode_tiles(x_bf16, H, S, S_in, S_pad, base3, base4, bidx, n_kv, kind, sm, codes, flags, slots, tile_bytes, head_start + H, stream)) return e;
  const int64_t ntiles = (S + T - 1) / T;
  return launch_overlapped(tile_scan_kernel, dim3((unsigned)H), SCAN_THREADS, (cudaStream_t)stream, ScanParams{{{tile_bytes, tile_off, head_bytes}, {}}, (int)ntiles, ntiles, head_start, total});
}

extern "C" int gaac_encode_begin(const void* x_bf16, int64_t H, int64_t S, int64_t S_in, int64_t S_pad,
                                 const uint8_t* base3, const uint8_t* base4, const int32_t* bidx, int n_kv, int kind,
                                 uint8_t* sm, uint8_t* codes, int32_t* flags, uint8_t* slots, int32_t* tile_bytes,
                                 int32_t* tile_off, int32_t* head_bytes, int32_t* head_start, void* stream) {
  return encode_begin(x_bf16, H, S, S_in, S_pad, base3, base4, bidx, n_kv, kind, sm, codes, flags, slots, tile_bytes, tile_off, head_bytes, head_start, nullptr, stream);
}

extern "C" int gaac_encode_queued(const void* x_bf16, int64_t H, int64_t S, int64_t S_in, int64_t S_pad,
                                  const uint8_t* base3, const uint8_t* base4, const int32_t* bidx, int n_kv, int kind,
                                  uint8_t* sm, uint8_t* codes, int32_t* flags, uint8_t* slots, int32_t* tile_bytes,
                                  int32_t* tile_off, int32_t* head_bytes, int32_t* head_start, int32_t* total_pinned, uint64_t* counter, void* stream) {
  if (!total_pinned || !counter || !tile_off || !head_bytes || !head_start) return GAAC_E_ARG;
  if (reinterpret_cast<uintptr_t>(counter) & 7) return GAAC_E_ALIGN;
  *reinterpret_cast<volatile int32_t*>(total_pinned) = -1;
  int e = encode_tiles(x_bf16, H, S, S_in, S_pad, base3, base4, bidx, n_kv, kind, sm, codes, flags, slots, tile_bytes, head_start + H, stream, reinterpret_cast<unsigned long long*>(counter), total_pinned);
  const int64_t ntiles = (S + T - 1) / T;
  if (!e) e = launch_overlapped(tile_scan_kernel, dim3((unsigned)H), SCAN_THREADS, (cudaStream_t)stream, ScanParams{{{tile_bytes, tile_off, head_bytes}, {}}, (int)ntiles, ntiles, head_start, nullptr});
  // The encode may be queued, since a launch also reports an error that an earlier call left behind, and then still writes *total_pinned, which goes with a failed call.
  if (e == GAAC_E_LAUNCH) { cudaStreamSynchronize((cudaStream_t)stream); cudaGetLastError(); }
  return e;
}

// The word is polled, since a wait for the stream would also wait for what was queued behind the kernel that writes it, and takes longer to return.  Now and then the stream is asked, which
// ends the wait when the kernels have failed.
extern "C" int gaac_wait_total(const int32_t* total_pinned, void* stream) {
  if (!total_pinned) return GAAC_E_ARG;
  const volatile int32_t* const word = total_pinned;
  while (true) {
    for (int i = 0; i < 4096; i++) {
      const int32_t total = *word;
      if (total != -1) { std::atomic_thread_fence(std::memory_order_acquire); return total >= 0 ? GAAC_OK : GAAC_E_ARG; }
      __builtin_ia32_pause();
    }
    const cudaError_t e = cudaStreamQuery((cudaStream_t)stream);
    if (e != cudaSuccess) cudaGetLastError();        // (reported here, so not by a later launch as well)
    if (e == cudaErrorNotReady) continue;
    return e == cudaSuccess && *word >= 0 ? GAAC_OK : GAAC_E_LAUNCH;
  }
}

extern "C" int gaac_encode_sized(const void* x_bf16, int64_t H, int64_t S, int64_t S_in, int64_t S_pad,
                                 const uint8_t* base3, const uint8_t* base4, const int32_t* bidx, int n_kv, int kind,
                                 uint8_t* sm, uint8_t* codes, int32_t* flags, uint8_t* slots, int32_t* tile_bytes,
                                 int32_t* tile_off, int32_t* head_bytes, int32_t* head_start, int32_t* total_pinned, void* stream) {
  if (!total_pinned) return GAAC_E_ARG;
  if (int e = encode_begin(x_bf16, H, S, S_in, S_pad, base3, base4, bidx, n_kv, kind, sm, codes, flags, slots, tile_bytes, tile_off, head_bytes, head_start, total_pinned, stream)) return e;
  return cudaStreamSynchronize((cudaStream_t)stream) == cudaSuccess ? GAAC_OK : GAAC_E_LAUNCH;
}

extern "C" int gaac_compact_copy(const uint8_t* slots, const int32_t* tile_bytes, int64_t H, int64_t ntiles, const int32_t* head_start, uint8_t* ovf,
                                 const int32_t* tile_off, int64_t tile_off_stride, const int32_t* flags, int64_t S, int64_t S_pad, int32_t* ovf_off,
                                 int zero_pad, int64_t ovf_cap, int64_t head_cap, int32_t* status, void* stream) {
  if (!slots || !tile_bytes || !head_start || !ovf || !tile_off || H <= 0 || ntiles <= 0 || tile_off_stride < ntiles || zero_pad < 0 || zero_pad > 32) return GAAC_E_ARG;
  if (ovf_cap < 0 || head_cap < 0 || H * ntiles > 0x7FFFFFF0LL) return GAAC_E_ARG;
  if (ovf_off && (!flags || S <= 0 || S_pad < S)) return GAAC_E_ARG;
  CompactParams p{};
  p.side[0] = CompactSide{slots, tile_bytes, tile_off, head_start, ovf, flags, ovf_off, status};
  p.ntiles = (int)ntiles; p.n_items = (unsigned)(H * ntiles); p.tile_off_stride = tile_off_stride; p.S = S; p.S_pad = S_pad;
  p.zero_pad = zero_pad; p.ovf_cap = ovf_cap; p.head_cap = head_cap;
  return launch_overlapped(compact_copy_kernel, compact_grid(p, 1), 128, (cudaStream_t)stream, p);
}

extern "C" int gaac_head_prefix(const int32_t* head_bytes, int64_t H, int32_t* head_start, void* stream) {
  if (!head_bytes || !head_start || H <= 0) return GAAC_E_ARG;
  head_prefix_kernel<<<1, SCAN_THREADS, 0, (cudaStream_t)stream>>>(head_bytes, (int)H, head_start);
  return launch_status();
}

extern "C" int gaac_decode_page(const uint8_t* sm, const uint8_t* codes, const int32_t* flags, const int32_t* tile_off, int64_t tile_off_stride,
                                const uint8_t* ovf, const int32_t* head_start, const uint8_t* base3, const uint8_t* base4, const int32_t* bidx,
                                int n_kv, int kind, int64_t H, int64_t S, int64_t S_pad, void* out_bf16, void* stream) {
  if (!sm || !codes || !flags || !tile_off || !ovf || !head_start || !base3 || !base4 || !out_bf16) return GAAC_E_ARG;
  if (H <= 0 || S <= 0 || S_pad < (S + T - 1) / T * T || S_pad % T || n_kv <= 0 || H > 65535 || (kind != GAAC_KIND_K && kind != GAAC_KIND_V)) return GAAC_E_ARG;
  if (!aligned16(sm) || !aligned16(codes) || !aligned16(out_bf16)) return GAAC_E_ALIGN;
  const int ntiles = (int)((S + T - 1) / T);
  const int per_warp = tiles_per_warp(ntiles, H, DEC_RESIDENT, DEC_MOST);
  const dim3 grid((ntiles + ENC_WARPS * per_warp - 1) / (ENC_WARPS * per_warp), (unsigned)H);
  return launch_overlapped(kind == GAAC_KIND_K ? decode_page_kernel<0> : decode_page_kernel<1>, grid, ENC_WARPS * 32, (cudaStream_t)stream, sm, codes, flags, tile_off, tile_off_stride, ovf,
                           head_start, base3, base4, bidx, n_kv, S, S_pad, (uint16_t*)out_bf16, ntiles, per_warp);
}

// a thread may read two channels at a time
static bool hist_pairs(const void* x, int64_t n_ch, int64_t row_stride) { return (reinterpret_cast<uintptr_t>(x) & 3) == 0 && n_ch % 2 == 0 && row_stride % 2 == 0; }
static dim3 hist_grid(int64_t n_ch, int64_t N, int kinds) { return dim3((unsigned)((n_ch + 127) / 128), (unsigned)((N + HIST_ROWS - 1) / HIST_ROWS), (unsigned)kinds); }

extern "C" int gaac_exponent_hist(const void* x_bf16, int64_t N, int64_t n_ch, long long* hist, void* stream) {
  if (!x_bf16 || !hist || N <= 0 || n_ch <= 0) return GAAC_E_ARG;
  // the grid's second dimension holds 65535 chunks: longer inputs take several launches
  constexpr int64_t MOST = 65535LL * HIST_ROWS;
  for (int64_t r = 0; r < N; r += MOST) {
    const int64_t rows = std::min(MOST, N - r);
    const HistParams<unsigned long long> p{{(const uint16_t*)x_bf16 + r * n_ch, nullptr}, {(unsigned long long*)hist, nullptr}, rows, n_ch, n_ch};
    if (hist_pairs(p.x[0], n_ch, n_ch)) exponent_hist_kernel<unsigned long long, true, false><<<hist_grid(n_ch, rows, 1), HIST_THREADS, 0, (cudaStream_t)stream>>>(p);
    else exponent_hist_kernel<unsigned long long, false, false><<<hist_grid(n_ch, rows, 1), HIST_THREADS, 0, (cudaStream_t)stream>>>(p);
  }
  return launch_status();
}

extern "C" int gaac_bases_from_hist(const long long* hist, int64_t n_rows, uint8_t* base3, uint8_t* base4, void* stream) {
  if (!hist || !base3 || !base4 || n_rows <= 0) return GAAC_E_ARG;
  const BasesParams<long long> p{{hist, nullptr}, {base3, nullptr}, {base4, nullptr}, n_rows, false};
  return launch_overlapped(bases_from_hist_kernel<long long>, dim3((unsigned)((n_rows + 3) / 4)), 128, (cudaStream_t)stream, p);
}

// ---------------------------------------------------------------------------------------------- slot cache: whole-prompt prefill
constexpr int CACHE_READ_PAD = 8;      // bytes kept free behind a head's escape bytes (the readers may touch them)

extern "C" size_t gaac_cache_calibrate_scratch_bytes(int n_kv) { return 2 * (size_t)(n_kv > 0 ? n_kv : 0) * D * 256 * sizeof(int32_t); }

// Histograms of both kinds, windows into the slot's rows of the tables.  zeroed: the counters are zero, and are left so, by a call that fails too; else they are cleared first,
// which takes a launch more.
template <class Cnt>
static int calibrate(const gaac_store* K, const gaac_store* V, const void* k_tok, const void* v_tok, int64_t L, int64_t row_stride, long n_ch, long at, uint8_t* counters, bool zeroed, cudaStream_t st) {
  Cnt* hist = reinterpret_cast<Cnt*>(counters);
  const long one = n_ch * PER_CHANNEL<Cnt>;
  const int n = (int)(2 * one * sizeof(Cnt) / 4);
  if (!zeroed) clear_kernel<<<std::min(n / 256, 8 * 148), 256, 0, st>>>(reinterpret_cast<u32*>(counters), n);
  const HistParams<Cnt> hp{{(const uint16_t*)k_tok, (const uint16_t*)v_tok}, {hist, hist + one}, L, n_ch, row_stride};
  const bool pairs = hist_pairs(k_tok, n_ch, row_stride) && hist_pairs(v_tok, n_ch, row_stride);
  const auto kernel = zeroed ? (pairs ? exponent_hist_kernel<Cnt, true, false> : exponent_hist_kernel<Cnt, false, false>) : (pairs ? exponent_hist_kernel<Cnt, true, true> : exponent_hist_kernel<Cnt, false, true>);
  int e = launch_overlapped(kernel, hist_grid(n_ch, L, 2), HIST_THREADS, st, hp);
  const BasesParams<Cnt> bp{{hist, hist + one}, {const_cast<uint8_t*>(K->base3) + at, const_cast<uint8_t*>(V->base3) + at},
                            {const_cast<uint8_t*>(K->base4) + at, const_cast<uint8_t*>(V->base4) + at}, n_ch, zeroed};
  if (!e) e = launch_overlapped(bases_from_hist_kernel<Cnt>, dim3((unsigned)((n_ch + 3) / 4), 2), 128, st, bp);
  if (e && zeroed) { cudaMemsetAsync(counters, 0, 4 * (size_t)n, st); cudaGetLastError(); }      // (the histogram may be queued: an error that an earlier call left behind is reported here too)
  return e;
}

extern "C" int gaac_cache_calibrate(const gaac_store* K, const gaac_store* V, const void* k_tok, const void* v_tok, int64_t L, int64_t row_stride, int slot, int n_kv,
                                    int n_base_rows, uint8_t* scratch, size_t scratch_bytes, void* stream) {
  if (!K || !V || !K->base3 || !K->base4 || !V->base3 || !V->base4 || !k_tok || !v_tok || !scratch) return GAAC_E_ARG;
  if (L <= 0 || L > 65535LL * HIST_ROWS || row_stride < (int64_t)n_kv * D || slot < 0 || n_kv <= 0 || n_kv > 256 || n_base_rows < (slot + 1) * n_kv) return GAAC_E_ARG;
  if (scratch_bytes < gaac_cache_calibrate_scratch_bytes(n_kv)) return GAAC_E_ARG;
  if (reinterpret_cast<uintptr_t>(scratch) & 3) return GAAC_E_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  const long n_ch = (long)n_kv * D, at = (long)slot * n_ch;
  return L <= 0xFFFF && aligned16(scratch) ? calibrate<Packed>(K, V, k_tok, v_tok, L, row_stride, n_ch, at, scratch, false, st)
                                           : calibrate<int>(K, V, k_tok, v_tok, L, row_stride, n_ch, at, scratch, false, st);
}

// Between the launches of a call its counters hold a prompt's counts, so the launches of another call with the same workspace must not come in between: the workspace's lock is
// held while they are queued (one of 64 by the address).
static std::mutex& workspace_lock(const void* workspace) {
  static std::mutex locks[64];
  return locks[(reinterpret_cast<uintptr_t>(workspace) >> 9) % 64];
}

extern "C" size_t gaac_cache_tables_workspace_bytes(int n_kv) { return n_kv > 0 ? 2 * (size_t)n_kv * D * 64 * sizeof(Packed) : 0; }

extern "C" int gaac_cache_prefill_own(const gaac_store* K, const gaac_store* V, const void* k_tok, const void* v_tok, int64_t L, int64_t row_stride, int slot, int n_kv,
                                      int32_t* tail_len, int32_t* seq_len, int64_t S_cap, int64_t ovf_cap, int n_base_rows, uint8_t* scratch, size_t scratch_bytes,
                                      int32_t* status, uint8_t* workspace, size_t workspace_bytes, void* stream) {
  if (!K || !V || !K->base3 || !K->base4 || !V->base3 || !V->base4 || !k_tok || !v_tok || !scratch || !workspace) return GAAC_E_ARG;
  if (L <= 0 || L > S_cap || row_stride < (int64_t)n_kv * D || slot < 0 || n_kv <= 0 || n_kv > 256 || n_base_rows < (slot + 1) * n_kv) return GAAC_E_ARG;
  if (scratch_bytes < gaac_cache_prefill_scratch_bytes(L, n_kv)) return GAAC_E_ARG;
  if (workspace_bytes < gaac_cache_tables_workspace_bytes(n_kv)) return GAAC_E_WORKSPACE;
  if (!aligned16(workspace)) return GAAC_E_ALIGN;
  if (L > 0xFFFF) {                                  // counts of 32 bits, in the scratch of the encode that follows (which has 2568 bytes for every 16 tokens of a head)
    if (int e = gaac_cache_calibrate(K, V, k_tok, v_tok, L, row_stride, slot, n_kv, n_base_rows, scratch, scratch_bytes, stream)) return e;
  } else {
    const long n_ch = (long)n_kv * D;
    const std::lock_guard<std::mutex> held(workspace_lock(workspace));
    if (int e = calibrate<Packed>(K, V, k_tok, v_tok, L, row_stride, n_ch, (long)slot * n_ch, workspace, true, (cudaStream_t)stream)) return e;
  }
  return gaac_cache_prefill(K, V, k_tok, v_tok, L, row_stride, slot, n_kv, tail_len, seq_len, S_cap, ovf_cap, n_base_rows, scratch, scratch_bytes, status, 0, stream);
}

static int clear_status(int32_t* status, cudaStream_t st) {           // the words that say whether an escape stream had room
  if (cudaMemsetAsync(status, 0, 4, st) == cudaSuccess && cudaMemsetAsync(status + 2, 0, 4, st) == cudaSuccess) return GAAC_OK;
  cudaGetLastError();
  return GAAC_E_LAUNCH;
}

extern "C" size_t gaac_cache_prefill_scratch_bytes(int64_t L, int n_kv) {
  const size_t items = (size_t)(L > 0 ? L / T : 0) * (size_t)(n_kv > 0 ? n_kv : 0);
  const size_t ctas = ((size_t)(L > 0 ? L / T : 0) + ENC_WARPS - 1) / ENC_WARPS * (size_t)(n_kv > 0 ? n_kv : 0);       // of the encoder, at most
  return 2 * items * (TILE_MAX_ESC + sizeof(int32_t)) + 2 * ctas * sizeof(int32_t) + 256;
}

extern "C" int gaac_cache_prefill(const gaac_store* K, const gaac_store* V, const void* k_tok, const void* v_tok, int64_t L, int64_t row_stride, int slot,
                                  int n_kv, int32_t* tail_len, int32_t* seq_len, int64_t S_cap, int64_t ovf_cap, int n_base_rows, uint8_t* scratch,
                                  size_t scratch_bytes, int32_t* status, int copy_only, void* stream) {
  if (!K || !V || !tail_len || !seq_len || !scratch || !status || (!copy_only && L > 0 && (!k_tok || !v_tok))) return GAAC_E_ARG;
  if (L < 0 || L > S_cap || S_cap % T || row_stride < (int64_t)n_kv * D || slot < 0 || n_kv <= 0 || n_kv > 256 || ovf_cap <= CACHE_READ_PAD ||
      n_base_rows <= 0 || n_base_rows % n_kv)
    return GAAC_E_ARG;
  for (const gaac_store* s : {K, V}) {
    if (!s->sm || !s->codes || !s->flags || !s->tile_off || !s->ovf || !s->ovf_used || !s->tail || !s->base3 || !s->base4) return GAAC_E_ARG;
    if (!aligned16(s->sm) || !aligned16(s->codes) || !aligned16(s->tail)) return GAAC_E_ALIGN;
  }
  if (!copy_only && (!aligned16(k_tok) || !aligned16(v_tok) || (row_stride * 2) % 16)) return GAAC_E_ALIGN;
  if (scratch_bytes < gaac_cache_prefill_scratch_bytes(L, n_kv)) return GAAC_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const long h0 = (long)slot * n_kv;
  const int ntiles = (int)(L / T);
  const long S = (long)ntiles * T, tiles_cap = S_cap / T, n_items = (long)n_kv * ntiles;
  if (n_items > 0x7FFFFFF0L) return GAAC_E_ARG;
  // Two launches for both kinds: encode, then offsets, copy, tails and counters; the encode clears the words that the
  // copy reports into.  scratch: escape slots of K, of V, then the tile sizes of K, of V, then those of the encoder's CTAs
  const gaac_store* side[2] = {K, V};
  const void* tok[2] = {k_tok, v_tok};
  EncodeParams ep{}; FinishParams fp{}; CompactParams cp{};
  ep.per_warp = tiles_per_warp(ntiles, 2 * n_kv, ENC_RESIDENT, ENC_MOST);
  const dim3 grid = encode_grid(ntiles, n_kv, 2, ep.per_warp);
  int32_t* const sizes = reinterpret_cast<int32_t*>(scratch + 2 * n_items * TILE_MAX_ESC);
  for (int kind = 0; kind < 2; kind++) {
    const gaac_store* s = side[kind];
    uint8_t* slots = scratch + kind * n_items * TILE_MAX_ESC;
    int32_t *tbytes = sizes + kind * n_items, *cbytes = sizes + 2 * n_items + (int64_t)kind * n_kv * grid.x, *toff = s->tile_off + h0 * tiles_cap;
    ep.side[kind] = EncodeSide{(const uint16_t*)tok[kind], s->base3 + (h0 % n_base_rows) * D, s->base4 + (h0 % n_base_rows) * D,          // consecutive heads, consecutive rows
                               s->sm + h0 * S_cap * D, s->codes + h0 * S_cap * CB, s->flags + h0 * S_cap, slots, tbytes, status + 2 * kind, cbytes, nullptr, nullptr};
    fp.side[kind] = FinishSide{slots, tbytes, cbytes, toff, s->ovf + h0 * ovf_cap, s->ovf_used + h0, status + 2 * kind, (const uint16_t*)tok[kind], (uint16_t*)s->tail + h0 * T * D};
    cp.side[kind] = CompactSide{slots, tbytes, toff, nullptr, s->ovf + h0 * ovf_cap, nullptr, nullptr, status + 2 * kind};
  }
  if (copy_only) {
    cp.ntiles = ntiles; cp.n_items = (unsigned)n_items; cp.tile_off_stride = tiles_cap; cp.head_stride = ovf_cap; cp.head_cap = ovf_cap - CACHE_READ_PAD;
    if (int e = clear_status(status, st)) return e;
    return ntiles ? launch_overlapped(compact_copy_kernel, compact_grid(cp, 2), 128, st, cp) : launch_status();
  }
  fp.L = L; fp.row_stride = row_stride; fp.tile_off_stride = tiles_cap; fp.ovf_cap = ovf_cap; fp.head_cap = ovf_cap - CACHE_READ_PAD; fp.n_kv = n_kv; fp.ntiles = ntiles;
  fp.per_cta = ENC_WARPS * ep.per_warp; fp.ctas = (int)grid.x; fp.chunk = FINISH_TILES / fp.per_cta * fp.per_cta; fp.chunks = (ntiles + fp.chunk - 1) / fp.chunk;
  fp.seq_len = seq_len + h0; fp.tail_len = tail_len + h0;
  if (ntiles) {
    ep.S = S; ep.x_head_stride = D; ep.x_row_stride = row_stride; ep.S_pad = S_cap; ep.n_kv = n_kv; ep.ntiles = ntiles;
    if (int e = launch_overlapped(encode_tiles_kernel<2>, grid, ENC_WARPS * 32, st, ep)) return e;
  }
  return launch_overlapped(prefill_finish_kernel, dim3((unsigned)(n_kv * fp.chunks + n_kv), 2), FINISH_THREADS, st, fp);
}
