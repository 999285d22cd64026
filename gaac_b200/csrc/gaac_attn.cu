// Fused decode attention over GAAC-compressed K/V (sm_100a): slot layout and paged layout in one kernel template.
//
// CTA = (batch row, kv head, context split), ATT_WARPS warps, one CTA per SM.  The CTA streams its 16-token tiles through one ring of
// shared-memory stages, each holding TPS consecutive tiles of K and V, filled by bulk asynchronous copies (the TMA engine without a
// tensor map, completion counted in bytes on the stage's mbarrier).  Warps take tiles from a shared counter, rebuild BF16 K/V fragments
// in registers (byte-SWAR) and feed mma.sync m16n8k16:
//   S^T[16 tok x 8 columns] = K[16 x 128] . Q^T        O^T[channel pairs x 8 columns] += V^T . P^T      (gaac_attn_tile.cuh)
// with an fp32 online softmax in the exp2 domain whose maximum is raised lazily.  Raw BF16 tiles (the slot layout's tail, the
// paged layout's filling block and raw-fallback tiles) are read straight from global memory into the same fragments.  The warps of a
// CTA are merged in shared memory, the CTA writes one partial (m, l, acc[128]) per query head, and the last CTA of a (row, kv head) to
// finish merges the splits and writes the output, so one launch does the whole layer.
//
// What the measurements on B200 say (they shaped the code below):
//  * the kernel is bound by the rebuild's instructions and by the latency that four warps per scheduler leave open, not by HBM (figures in gaac_attn_tile.cuh).  With a
//    private two-stage ring per warp every warp issued eight copies per tile pair, about 200 of 1354 instructions; one copy of four tiles, issued by the warp that is
//    last to leave a stage, takes that to about 25 per tile pair.
//  * a bulk copy takes the warp that issues it about 100 cycles, and a loop over the lanes before it where its operands are not known to be uniform: the
//    eight copies of a stage took their warp 2300 cycles, issued by an elected lane of the converged warp 1150 (57.5 -> 56.7 us at 65536 tokens).
//  * warps of their own for parts of the work lose: one that issues all copies is too slow by itself (56.3 us, but 620 instead of 500 on paged tiles), and with
//    four, six or eight of the sixteen warps expanding escape bytes (plan_tile, one tile or a whole stage at a time) the others wait for them: 65 to 88 us.
//  * bulk copies want few large copies (one 128-byte copy per row, which would allow a conflict-free skewed layout, was 15 % slower), so
//    shared memory holds the storage order and the 16-byte fragment reads accept a 2-way bank conflict, which costs nothing: a build that read other bytes without
//    conflicts, for timing only, took the same 51.3 us.
//
// Fragment conventions follow the reference kernel (gaac/kernel.py:62-66,160-194), whose storage order they mirror.
#include <algorithm>
#include <atomic>
#include "gaac_api.cuh"
#include "gaac_attn_tile.cuh"

namespace gaac {

// Warps per CTA (18 or 20 warps at 96 registers: 64.5 us instead of 57.5 at 65536 tokens; with the queries in shared memory, so that they spill 28 bytes only, 58.1 and 58.8 instead of 55.3).
constexpr int ATT_WARPS = 16, ATT_THREADS = ATT_WARPS * 32;
// ---- ring of stages.  A stage holds TPS consecutive tiles.
//   slot layout:  per side  sign/mantissa of the tiles (TPS x 2048) | codes (TPS x 768) | tag words (TPS x 64) | the tiles' escape bytes, which are
//                 contiguous in memory: one window of at most SIDE_ESC bytes that starts at the 16-byte boundary below the first
//   paged layout: TPS x {K slot, V slot}, each as it lies in the block buffer (one copy per slot, at most PSLOT bytes of it)
// Four tiles per stage: eight copies of 256 B .. 8 KB per four tile pairs; eight stages keep sixteen tiles in flight behind the sixteen in use.
constexpr int TPS = 4, NSTG = 8;
constexpr int SIDE_ESC = TPS * (ESC_WIN + 16);
constexpr int SB_CD = TPS * TILE_SM, SB_FL = SB_CD + TPS * TILE_CD, SB_ESC = SB_FL + TPS * 4 * T, SIDE_BYTES = SB_ESC + SIDE_ESC;
constexpr int STAGE_BYTES = 2 * SIDE_BYTES;
static_assert(SIDE_BYTES == TPS * PSLOT, "both layouts use stages of the same size");
// CTA tables: addend and segment table, K / V base words; per stage the mbarrier that counts arriving bytes and how many tiles of it the warps have left so far; per
// tile of a stage {address of its escape bytes of K, how many are staged, the same of V}, its metadata, and the word (stage + 1) << 4 | bits 2, 3: the K / V tile is
// raw, by which a warp knows the use of the slot: a parity can be two phases off for one that runs ahead of a slow one.  Then the metadata of the tiles that come next into the stage
// (and of the one behind them), which the warp that has the stage's last tile asks for and leaves there for the one that is last to leave the stage: asked for by each of the four in case that it
// is the one, they cost 10 instructions per tile pair more (64 x 32768 198.8 -> 196.0 us, paged 16 x 4096..65536 404 -> 398, 65536 tokens 49.4 -> 49.2).  Then the warps' segment areas.
constexpr int TB_BASES = ADDEND_BYTES + SEGTAB_BYTES, TB_FULL = TB_BASES + PAIR_BASES_BYTES, TB_LEFT = TB_FULL + 8 * NSTG, TB_ESC = TB_LEFT + 4 * NSTG, TB_META = TB_ESC + 16 * TPS * NSTG,
              TB_USE = TB_META + 8 * TPS * NSTG, TB_NEXT = TB_USE + 4 * TPS * NSTG, TB_AREA = TB_NEXT + 8 * (TPS + 1) * NSTG, TB_RING = TB_AREA + ATT_WARPS * AREA_BYTES;
constexpr int ATT_SMEM = TB_RING + NSTG * STAGE_BYTES + 16;          // (an escape segment is read as whole words)
static_assert(TB_BASES % 16 == 0 && TB_ESC % 16 == 0 && TB_AREA % 16 == 0 && TB_RING % 16 == 0 && STAGE_BYTES % 16 == 0 && SIDE_BYTES % 16 == 0 && SB_ESC % 16 == 0 && SB_FL % 16 == 0 && PSLOT % 16 == 0 && TB_FULL % 8 == 0 && SIDE_ESC % 16 == 0,
              "bulk copies need 16-byte aligned shared-memory destinations and sizes");
static_assert(ATT_SMEM + 368 <= 232448, "one CTA per SM: at most 227 KB of shared memory, static part included");
static_assert(ATT_THREADS / 128 * 2 >= 8, "the fused exchange keeps at most two merged heads per thread");
constexpr int ACC_LD = D + 8;                        // row stride of the staged accumulators: 8j + r banks, conflict-free stores

struct AttnParams {
  // slot layout
  gaac_side K, V;
  const int* slot; const int* seq_len; const int* tail_len; int tail_cap; long S_pad; int n_base_rows;
  int S_uniform;                 // tokens of every cache head when seq_len == NULL (slot == NULL: batch row b reads slot b)
  // paged layout
  const uint8_t* buf; const uint16_t* raw; const int* mt; const int* bt; long bt_stride; int TS; int ovf_slot;
  const uint8_t *b3k, *b4k, *b3v, *b4v;
  // common
  const uint16_t* q; int B, n_q, n_kv, G; float scale_log2; int nsplit;
  int* counters; int* err; float* pm; float* pl; float* pa;     // err: set to 1 when a bounded wait inside the kernel ran out
  uint16_t* out; float* out_f32; float* part;
  // balanced launches (units > 0; grid = (n_kv, units)): the rows share `units` ranges per kv head by their lengths, see row_share; nsplit is not used, a
  // unit of a kv head has one partial per query head, at (kvh * units + unit) * G
  int units, wave;                                  // wave: units of a kv head that run at a time
  int flat;                                         // flat launches: CTAs (0: not one); nsplit is not used, see FlatWalk
  // cross-GPU exchange (x_recv == NULL: unused): the partial of every query head is stored into every rank's receive
  // buffer, then this rank's arrival flag of the (row, kv head) group on every rank is set to the exchange number; with
  // x_fused the same CTA then waits (bounded) for the other ranks' flags, merges all ranks' rows and writes the output
  const int2* row_order;                            // paged layout, optional: {batch row, its token count}, longest row first
  int2* order_buf;                                  // room for B entries of it in the workspace
  unsigned long long* const* x_recv; int* x_epoch; int* x_ticket; int* x_err; int x_rank, x_world, x_rows_cap, x_fused;
  // debug instantiation only: the rebuilt BF16 K / V rows are written to [B*n_kv, dump_S, 128] (row = token of the head)
  uint16_t* dump_k; uint16_t* dump_v; long dump_S;
};

// ---- cross-GPU exchange helpers.  A receive buffer holds 8-byte entries: the low word is an fp32 value, the high word the
// number of the exchange it belongs to.  An entry is written with ONE 64-bit store and read with one 64-bit load, so a reader
// that sees the right number has the value that came with it: no flag, no fence and no second trip over NVLink is needed to
// know that a row has arrived.  Every wait is bounded: after X_WAIT_LIMIT polls (about a second) the reader gives up, so a
// missing peer never hangs the GPU.
constexpr int X_WAIT_LIMIT = 1000000;
__device__ __forceinline__ void x_store(unsigned long long* p, float v, u32 tag) {
  const unsigned long long e = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
  asm volatile("st.relaxed.sys.global.b64 [%0], %1;" ::"l"(p), "l"(e) : "memory");
}
__device__ __forceinline__ bool x_load(const unsigned long long* p, u32 tag, float& v) {
  for (int it = 0; it < X_WAIT_LIMIT; it++) {
    unsigned long long e;
    asm volatile("ld.relaxed.sys.global.b64 %0, [%1];" : "=l"(e) : "l"(p) : "memory");
    if ((u32)(e >> 32) == tag) { v = __uint_as_float((u32)e); return true; }
    if (it > 64) __nanosleep(100);
  }
  v = 0.f;
  return false;
}
// Wait for and merge the rows of all ranks for query head qh, element d: base = this exchange's half of the receive buffer,
// [world][rows_cap][130] entries of (m in natural-log units, l, acc[128]); same algebra as the split merge.  Returns false when
// a row did not arrive in time.
__device__ __forceinline__ bool x_merge_rows(const unsigned long long* base, int world, long rows_cap, long qh, int d, u32 tag, float& out) {
  float M = -CUDART_INF_F;
  bool ok = true;
  for (int s = 0; s < world && ok; s++) { float m; ok = x_load(base + (s * rows_cap + qh) * 130, tag, m); M = fmaxf(M, m); }   // one bound in all: stop at the first row that does not come
  float L = 0.f, Ac = 0.f;
  for (int s = 0; s < world && ok; s++) {
    const unsigned long long* pp = base + (s * rows_cap + qh) * 130;
    float ms, l, a;
    ok &= x_load(pp, tag, ms) & x_load(pp + 1, tag, l) & x_load(pp + 2 + d, tag, a);
    const float f = (ms == -CUDART_INF_F) ? 0.f : __expf(ms - M);
    L += l * f; Ac += a * f;
  }
  out = (ok && L > 0.f) ? Ac / L : 0.f;
  return ok;
}

// ---- merge of the splits.  The ticket is taken with an acquire-release atomic at GPU scope by one thread between two CTA barriers: the
// barrier before it orders every thread's partial stores before the release, the barrier after it orders the acquire before every
// thread's loads of the other CTAs' partials - no per-thread fence is needed.
__device__ __forceinline__ bool last_split(int* counter, int NS, int* s_last) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int ticket;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(ticket) : "l"(counter) : "memory");
    *s_last = (ticket == NS - 1);
    if (ticket == NS - 1) *counter = 0;               // leave the counter ready for the next call
  }
  __syncthreads();
  return *s_last != 0;
}
// Partials of a head, that of split s at first + s * step -> M, L and element d of the sum, by the whole warp.  A lane has the weights of one split, so nothing but
// shuffles passes between the loads of up to 32 splits, which are all in flight at once, and the result.  (With a split per warp, weights and sums through shared memory and the
// splits beyond 16 loaded behind the others, the CTA that is last took 2.1 us at 18 splits, 1.9 at 8; now 1.4.)
template <int N> __device__ __forceinline__ void merge_splits(const AttnParams& p, long first, int step, int NS, int d, float& M, float& L, float& acc) {
  const int lane = threadIdx.x & 31;
  M = -CUDART_INF_F; L = 0.f; acc = 0.f;
#pragma unroll 1
  for (int s0 = 0; s0 < NS; s0 += N) {
    const int n = min(N, NS - s0);
    const long at = first + (long)s0 * step;
    const float* v0 = p.pa + at * D + d;
    float v[N];
#pragma unroll
    for (int k = 0; k < N; k += 8)
      if (k < n) {
#pragma unroll
        for (int s = k; s < k + 8; s++) v[s] = __ldcg(v0 + (long)min(s, n - 1) * step * D);
      }
    const float m = lane < n ? __ldcg(p.pm + at + (long)lane * step) : -CUDART_INF_F, l = lane < n ? __ldcg(p.pl + at + (long)lane * step) : 0.f;
    float most = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(FULLM, most, o));
    most = fmaxf(most, M);
    const float keep = M == -CUDART_INF_F ? 0.f : fast_exp2(M - most), f = m == -CUDART_INF_F ? 0.f : fast_exp2(m - most);
    float sum = l * f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULLM, sum, o);
    M = most; L = L * keep + sum; acc *= keep;
#pragma unroll
    for (int k = 0; k < N; k += 8)
      if (k < n) {
#pragma unroll
        for (int s = k; s < k + 8; s++) {
          const float w = __shfl_sync(FULLM, f, s);
          if (s < n) acc += w * v[s];                // (an infinite value and a weight of zero make NaN)
        }
      }
  }
}

// The same of `heads` heads (heads <= HMAX <= 8), that of head g and split s at first + g * per_head + s * per_split -> deliver(head, M, L, acc[threadIdx.x & 127]), through shared memory: the
// flat launches' loop over pieces leaves no registers for the form above (64 x 32768 tokens, groups of 8: 220 us with it and 100 bytes of spills, 210 with this), and their pairs have few pieces.
template <int HMAX, class F>
__device__ __forceinline__ void merge_pieces(const AttnParams& p, uint8_t* area, long first, int per_head, int per_split, int heads, int NS, const F& deliver) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* c_f = reinterpret_cast<float*>(area);        // [heads][NS]  m, then exp2(m - M)
  float* c_l = c_f + 8 * NS;                          // [heads][NS]  l
  float* c_ML = c_l + 8 * NS;                         // [8][2]       M, L per head
  float* c_red = c_ML + 16;                           // [W][8][128]  (NS <= 1024 keeps this inside the ring area)
  for (int i = tid; i < heads * NS; i += ATT_THREADS) {
    const long at = first + (per_split == 1 ? i : i / NS * per_head + i % NS * per_split);          // (per_split 1: NS places per head)
    c_f[i] = __ldcg(p.pm + at); c_l[i] = __ldcg(p.pl + at);
  }
  float4 acc[HMAX];                                   // split `warp` of every head, in flight while M and L are computed
#pragma unroll
  for (int g = 0; g < HMAX; g++)
    acc[g] = (g < heads && warp < NS) ? __ldcg(reinterpret_cast<const float4*>(p.pa + (first + g * per_head + warp * per_split) * D) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  if (warp < heads) {
    float M = -CUDART_INF_F;
    for (int s2 = lane; s2 < NS; s2 += 32) M = fmaxf(M, c_f[warp * NS + s2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(FULLM, M, o));
    float L = 0.f;
    for (int s2 = lane; s2 < NS; s2 += 32) {
      const float ms = c_f[warp * NS + s2];
      const float f = (ms == -CUDART_INF_F) ? 0.f : fast_exp2(ms - M);
      c_f[warp * NS + s2] = f; L += c_l[warp * NS + s2] * f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(FULLM, L, o);
    if (lane == 0) { c_ML[2 * warp] = M; c_ML[2 * warp + 1] = L; }
  }
  __syncthreads();
#pragma unroll
  for (int g = 0; g < HMAX; g++) {
    const float f = (g < heads && warp < NS) ? c_f[g * NS + warp] : 0.f;
    acc[g] = make_float4(acc[g].x * f, acc[g].y * f, acc[g].z * f, acc[g].w * f);
  }
  for (int s2 = warp + ATT_WARPS; s2 < NS; s2 += ATT_WARPS) {
#pragma unroll
    for (int g = 0; g < HMAX; g++) {
      if (g < heads) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p.pa + (first + g * per_head + s2 * per_split) * D) + lane);
        const float f = c_f[g * NS + s2];
        acc[g].x += v.x * f; acc[g].y += v.y * f; acc[g].z += v.z * f; acc[g].w += v.w * f;
      }
    }
  }
#pragma unroll
  for (int g = 0; g < HMAX; g++)
    if (g < heads) *reinterpret_cast<float4*>(c_red + ((warp * 8 + g) * D) + 4 * lane) = acc[g];
  __syncthreads();
  for (int g = tid >> 7; g < heads; g += ATT_THREADS / 128) {
    float Ac = 0.f;
    const int d = tid & 127;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; w++) Ac += c_red[(w * 8 + g) * D + d];
    deliver(g, c_ML[2 * g], c_ML[2 * g + 1], Ac);
  }
}

// Balanced launches: lane = batch row, tiles = the row's tiles.  Every row gets ceil(tiles / C) ranges (at least one, so that an empty row is written
// too), with the smallest C of at least SHARE_MIN_TILES for which all of them fit into the units there are; a few steps of bisection between the bounds
// total / units and total / (units - rows), which always fits.  Unit u then is range `split` of NS of row `row`; row >= 32: nothing to do.
// A ragged batch split alike for every row waits for its longest row.  `wave` units run at a time; of a launch with more, those behind the first
// wave are used only where that is faster: few units per row may leave much of the first wave idle (7 equal rows get 2 of 18 units each, in two waves 5
// of 37).  A second wave costs a prologue, about as long as 40 tiles; CTAs that find nothing to do cost 12.
constexpr int SHARE_MAX_ROWS = 32, SHARE_MIN_TILES = 4, SHARE_WAVE_TILES = 40 - 12;
__device__ __forceinline__ void row_share(int tiles, int B, int units, int wave, int u, int lane, int& row, int& split, int& NS) {
  const unsigned n = lane < B ? (unsigned)max(tiles, 0) : 0u, total = __reduce_add_sync(FULLM, n), most = __reduce_max_sync(FULLM, n);
  auto smallest = [&](int units) {
    unsigned lo = max((unsigned)SHARE_MIN_TILES, (total + units - 1) / units);
    unsigned hi = max(lo, units > B ? (total + (units - B) - 1) / (units - B) : most);
#pragma unroll 1
    for (int it = 0; it < 6 && lo < hi; it++) {
      const unsigned mid = (lo + hi) >> 1, want = lane < B ? max(1u, (n + mid - 1) / mid) : 0u;
      if (__reduce_add_sync(FULLM, want) <= (unsigned)units) hi = mid; else lo = mid + 1;
    }
    return hi;
  };
  unsigned hi = smallest(min(units, wave));
  if (units > wave) {
    const unsigned two = smallest(units);
    if (hi > SHARE_WAVE_TILES + 2 * two) hi = two;
  }
  const int ns = lane < B ? (int)max(1u, (n + hi - 1) / hi) : 0;
  u32 inc = (u32)ns;
  scan_step(inc, 1); scan_step(inc, 2); scan_step(inc, 4); scan_step(inc, 8); scan_step(inc, 16);
  row = popc(__ballot_sync(FULLM, (int)inc <= u));
  NS = __shfl_sync(FULLM, ns, row & 31);
  split = u - ((int)__shfl_sync(FULLM, inc, row & 31) - NS);
}

// Weights of a warp summed over its lanes; true when some sum of values is not finite although its weights are (see sum_exact).
template <int NSET> __device__ __forceinline__ bool sum_warp(WarpAcc<NSET>& A) {
  bool bad = false;
#pragma unroll
  for (int s = 0; s < NSET; s++) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) A.l[s] += __shfl_xor_sync(FULLM, A.l[s], o);
    u32 most = 0u;
#pragma unroll
    for (int i = 0; i < 16; i++) most = max(most, __float_as_uint(A.acc[s][i >> 2][i & 3]) & 0x7FFFFFFFu);
    bad |= most >= 0x7F800000u && A.l[s] < CUDART_INF_F;
  }
  return bad;
}
// A warp's sums on their way into the CTA's: m [W][8], l [W][8], acc [W][8][ACC_LD]
template <int NSET> __device__ __forceinline__ void stage_warp(const WarpAcc<NSET>& A, uint8_t* area, int G, int warp, int lane) {
  const int j = lane & 3, r = lane >> 2;
  float* sh_m = reinterpret_cast<float*>(area);
#pragma unroll
  for (int s = 0; s < NSET; s++) {
    const int h = 4 * s + j;
    if (r == 0) { sh_m[warp * 8 + h] = A.m[s]; sh_m[ATT_WARPS * 8 + warp * 8 + h] = A.l[s]; }
    if (h < G) {
      float* a0 = sh_m + ATT_WARPS * 16 + (warp * 8 + h) * ACC_LD + r;
#pragma unroll
      for (int i = 0; i < 16; i++) a0[8 * acc_channel(i >> 2, i & 3)] = A.acc[s][i >> 2][i & 3];
    }
  }
}
static_assert(ATT_THREADS == 512, "a thread of the merge has every fourth head");
// Head g of the warps w0, w0 + step, .. (N of them), as they left it in shared memory (m [W][8], l [W][8], acc [W][8][ACC_LD]) -> M, L and element d of the
// sum
// (A lane has the weight of one warp: with all of them by every thread, 48 loads from shared memory instead of 18, the CTA took 0.2 us more.)
template <int N> __device__ __forceinline__ void merge_warps(const uint8_t* area, int step, int w0, int g, int d, float& M, float& L, float& acc) {
  const float *sh_m = reinterpret_cast<const float*>(area), *sh_l = sh_m + ATT_WARPS * 8, *sh_acc = sh_l + ATT_WARPS * 8;
  const int own = (step * (threadIdx.x % N) + w0) * 8 + g;
  const float m = sh_m[own], l = sh_l[own];
  M = m;
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(FULLM, M, o));
  const float f = m == -CUDART_INF_F ? 0.f : fast_exp2(m - M);
  L = l * f; acc = 0.f;
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1) L += __shfl_xor_sync(FULLM, L, o);
#pragma unroll
  for (int w = 0; w < N; w++) acc += sh_acc[((step * w + w0) * 8 + g) * ACC_LD + d] * __shfl_sync(FULLM, f, w);
}
// ---- V elements that are not finite.  In the value product of groups up to 4 a word meets a weight of zero for the other parity's channel, and the lower
// half of a weight may be zero or negative in any group: an infinite or NaN element makes its word's OTHER channel NaN as well (0 x Inf), and its own NaN where Inf is
// right.  A CTA whose sum is not finite therefore takes its range once more in plain fp32, where an element meets its own weight only and tokens
// behind the end meet none: range `split` of NS of (row, kv head) bh, straight from global memory, token by token, four channels per lane.  The
// result lies where the warps of the main loop leave theirs.  Finite data never comes here, and what counts is what the presence of this code costs
// the main loop: it looks everything up again and has little code and few registers.  32768 tokens, 8 kv heads: finite 33.8 -> 33.5 us, one infinite
// element 608; head_dim 256: finite 36.1 -> 36.5.  With the main loop's decoder in its place a second pass took a fifth of that, but finite data
// 1 to 7 % more, inlined or called.
template <bool PAGED, bool WIDE>
__device__ __forceinline__ void sum_exact(const AttnParams& p, uint8_t* area, int bh, int split, int NS, const int* range = nullptr) {
  int tid = threadIdx.x;
  asm volatile("" : "+r"(tid), "+r"(bh), "+r"(split), "+r"(NS));
  const int lane = tid & 31, warp = tid >> 5, b = bh / p.n_kv, kvh = bh % p.n_kv, hf = WIDE ? warp & 1 : 0, HALVES = WIDE ? 2 : 1;
  int S, ch = 0, TL = 0;
  if (PAGED) S = p.seq_len[b];
  else {
    const int sl = p.slot ? p.slot[b] : b;
    ch = max(sl, 0) * p.n_kv + kvh;
    S = sl < 0 ? 0 : p.seq_len ? p.seq_len[ch] : p.S_uniform;
    TL = sl >= 0 && p.tail_len && split == NS - 1 ? p.tail_len[ch] : 0;
  }
  const int ntiles = (S + 15) >> 4, chunk = (ntiles + NS - 1) / NS, tlo = range ? min(range[0], ntiles) : min(split * chunk, ntiles);
  const int n = range ? (split == NS - 1 ? ntiles - tlo : min(range[1], ntiles - tlo)) : min(chunk, ntiles - tlo);                  // (as the main loop takes it)
  float m[8], l[8], acc[8][4];
#pragma unroll
  for (int h = 0; h < 8; h++) { m[h] = -CUDART_INF_F; l[h] = acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f; }
#pragma unroll 1
  for (int i = WIDE ? warp >> 1 : warp; i < n + ((TL + T - 1) >> 4); i += ATT_WARPS / HALVES) {
    const int tile = tlo + i, valid = i < n ? min(T, S - tile * T) : min(T, TL - (i - n) * T);
    PlainSide side[3];                               // K (of both halves where there are two), V
    u32 tags[3]; int at[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (!WIDE && c == 1) continue;
      const bool vs = c == 2;
      PlainSide& s = side[c];
      const uint8_t* fl;
      if (PAGED) {
        const int t = 2 * (HALVES * kvh + (vs ? hf : c)) + (vs ? 1 : 0), row = (t >> 1) * D, meta = p.mt[p.bt[(long)b * p.bt_stride + tile] * (2 * HALVES * p.n_kv) + t];
        const uint8_t* t0 = p.buf + (long)meta * p.TS;
        s = PlainSide{t0, t0 + SLOT_CD_OFF, t0 + SLOT_OVF_OFF, (vs ? p.b3v : p.b3k) + row, (vs ? p.b4v : p.b4k) + row, meta < 0 ? p.raw + (long)raw_tile(meta) * (T * D) : nullptr};
        fl = t0 + SLOT_FL_OFF;
      } else {
        const gaac_side& g = vs ? p.V : p.K;
        const long row = (long)ch * p.S_pad + (long)tile * T;
        const int brow = ch % p.n_base_rows * D;
        s = PlainSide{g.sm + row * D, g.codes + row * CB, nullptr, g.base3 + brow, g.base4 + brow, nullptr};
        if (i < n) s.esc = g.ovf + ((long)g.head_start[ch] + g.tile_off[(long)ch * (p.S_pad >> 4) + tile]);
        else s.raw = reinterpret_cast<const uint16_t*>(g.tail) + ((long)ch * p.tail_cap + (i - n) * T) * D;
        fl = reinterpret_cast<const uint8_t*>(g.flags + row);
      }
      tags[c] = s.raw ? 0u : reinterpret_cast<const u32*>(fl)[lane & 15];
      const u32 own = (u32)row_esc_bytes(tags[c]);
      u32 inc = own;
      scan_step(inc, 1); scan_step(inc, 2); scan_step(inc, 4); scan_step(inc, 8);
      at[c] = (int)(inc - own);
    }
#pragma unroll 1
    for (int tok = 0; tok < valid; tok++) {
      float sc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < (WIDE ? 2 : 1); c++) {
        const u32 tg = __shfl_sync(FULLM, tags[c], tok);
        const int ea = __shfl_sync(FULLM, at[c], tok);
#pragma unroll 1
        for (int d = lane; d < D; d += 32) {
          const float x = plain_element<false>(side[c], tok, d, tg, ea);
#pragma unroll
          for (int h = 0; h < 8; h++)
            if (h < p.G) sc[h] += x * __uint_as_float((u32)p.q[(((long)b * p.n_q + kvh * p.G + h) * HALVES + c) * D + d] << 16);
        }
      }
      const u32 tg = __shfl_sync(FULLM, tags[2], tok);
      const int ea = __shfl_sync(FULLM, at[2], tok);
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) v[q] = plain_element<true>(side[2], tok, lane + 32 * q, tg, ea);
#pragma unroll
      for (int h = 0; h < 8; h++) {
        float s = sc[h];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULLM, s, o);
        s *= p.scale_log2;
        if (s > m[h]) {
          const float f = fast_exp2(m[h] - s);
          l[h] *= f; m[h] = s;
#pragma unroll
          for (int q = 0; q < 4; q++) acc[h][q] *= f;
        }
        const float w = fast_exp2(s - fmaxf(m[h], -1e30f));
        l[h] += w;
#pragma unroll
        for (int q = 0; q < 4; q++) acc[h][q] += w * v[q];
      }
    }
  }
  float* sh_m = reinterpret_cast<float*>(area);
#pragma unroll
  for (int h = 0; h < 8; h++) {
    if (lane == 0) { sh_m[warp * 8 + h] = m[h]; sh_m[ATT_WARPS * 8 + warp * 8 + h] = l[h]; }
#pragma unroll
    for (int q = 0; q < 4; q++) sh_m[ATT_WARPS * 16 + (warp * 8 + h) * ACC_LD + lane + 32 * q] = acc[h][q];
  }
}

// ---- flat launches: one wave of CTAs shares the (row, kv head) pairs; every CTA sees the lengths and makes the same plan, one of three.  A piece of a pair costs its CTA
// about as much as FLAT_EXTRA tiles beside its own (tables of the bases, queries, first copies, merges).
//  line    all pairs one behind the other, FLAT_EXTRA places in front of each, every CTA an equal share of the places: CTA c has [c * share, (c + 1) * share).  An
//          empty pair (its output is zero) goes to the CTA that has its last place.  A CTA begins in the middle of a pair and pays for that piece: share + FLAT_EXTRA.
//  single  no more pairs than CTAs: every pair in ceil(tiles / C) equal pieces (or in as many as every other, where they are about equally long), one piece per CTA, where
//          the smallest C for which the CTAs suffice is no more than share (and SLACK).
//  whole   more pairs than CTAs: the pairs in order of length, longest first, dealt out forth and back.  Where the CTA that gets most has no more than the line's, it saves the
//          pieces in the middle and the merges.  That is what short rows want, and a caller who has a table (or a capacity) much wider than its rows are long.
// A piece has its partials at (CTA + pair) * G, which no two pieces share: pieces of a pair are those of consecutive CTAs, in order.
// A grid of several waves pays a prologue, the merges and the wait for its slowest CTA with every wave, about 8.5 us, and half a wave is as dear as a whole one.
// us, grid -> flat: 16 rows x 8 kv heads of 4K-64K tokens 452 -> 403, 64 x 1 of 32K (groups of 8) 219 -> 202, 8 x 8 of 4K-16K 89 -> 77 (a balanced launch before).
// The line alone, and now: 64 x 8 of 100-400 in a table of 8192 39.9 -> 32.0, 32 x 8 of 20-2000 49.1 -> 42.2, 24 x 8 of 64-600 23.9 -> 16.7, 512 x 1 of 50-600 48.4 -> 38.7, 8 x 8 of 200-3000
// 18.4 -> 15.7, 37 x 4 of 8K 113.8 -> 108.0, 300 x 1 of 100-2000 67.3 -> 66.6;  head_dim 256: 32 x 8 of up to 1000 53.8 -> 40.1, 8 x 4 of 100-700 15.1 -> 13.2.
// FLAT_EXTRA 24 / 36 / 48 (of the line): 16 x 8 421 / 422 / 424, 12 x 8 of 500-6000 - / 43.0 / 44.5, 64 x 1 - / 218 / 216.
// A tile of head_dim 256 is twice the work: with 18 there, 36 -> 18, 32 x 4 of 200-2000 43.4 -> 37.9, 16 x 8 of 1K-8K 125.0 -> 118.3, 20 x 8 of 200-3000 69.9 -> 63.1, 9 x 4 of 4K-30K 108.3 -> 106.5, 6 x 8
// of 1K-16K (groups of 8) 81.3 -> 80.0, 8 x 4 of 1K-8K the same; 24 118 -> 120 and 63 -> 66, 14 up to 2.5 % slower in groups of 8.  FLAT_SLACK, what a piece of `single` may have beyond share, since the
// line's pieces in the middle are dearer than share too: without it 16 x 8 of 2000 56.4 -> 58.7, with 18 12 x 4 of 2K-20K 104.4 -> 108.0.  At head_dim 128 42 in place of 36 and 21 for the slack: 64 x 1
// slots 190.0 -> 187.7, 12 x 8 of 500-6000 38.8 -> 40.6, others the same: left.
constexpr int FLAT_EXTRA = 36, FLAT_SLACK = 0, FLAT_EXTRA256 = 18, FLAT_SLACK256 = 9;
constexpr int FLAT_ROWS = 2048, FLAT_SORT = ATT_THREADS, FLAT_WHOLE = 32;               // rows whose tiles are held while the plan is made; rows that are sorted; pairs of a CTA that are dealt out
constexpr int FLAT_SCRATCH = 4 * (FLAT_ROWS + 2 * FLAT_SORT + 4 * ATT_WARPS);
struct FlatWalk {
  int share, lo, hi;                                  // of the CTA, on the line; share 0: single, below zero: whole
  int row, kvh, at, tiles;                            // the pair that is looked at next: its first place on the line, its tiles; single, whole: `at` pieces are left
  int pair, range[2], split, ns, tokens;              // the piece found: pair = row * n_kv + kvh (below zero: no more), its first tile and how many, which of the pair's pieces; the row's tokens
};
__device__ __forceinline__ int tiles_in(int tokens) { return max((tokens + 15) >> 4, 0); }
// Executed by the whole CTA; warp 0 gets the walk.  window: 64 words for flat_next;  scratch: FLAT_SCRATCH bytes that are free until the first piece begins;  least: tiles
// of a piece of `single`, at least.
template <int EXTRA, int SLACK, class F> __device__ __forceinline__ void flat_plan(FlatWalk& f, int B, int n_kv, int least, int* window, int* scratch, const F& tokens_of) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, ctas = gridDim.x, pairs = B * n_kv;
  int* const held = scratch;                          // the rows' tokens
  int* const order = held + FLAT_ROWS;
  int* const keys = order + FLAT_SORT;
  u32* const red = reinterpret_cast<u32*>(keys + FLAT_SORT);
  u32 sum = 0u, longest = 0u, shortest = 0xFFFFFFFFu;
  for (int r = tid; r < B; r += ATT_THREADS) {
    const int tokens = tokens_of(r);
    const u32 t = (u32)tiles_in(tokens);
    if (r < FLAT_ROWS) held[r] = tokens;
    sum += t; longest = max(longest, t); shortest = min(shortest, t);
  }
  sum = __reduce_add_sync(FULLM, sum); longest = __reduce_max_sync(FULLM, longest); shortest = __reduce_min_sync(FULLM, shortest);
  if (lane == 0) { red[warp] = sum; red[ATT_WARPS + warp] = longest; red[2 * ATT_WARPS + warp] = shortest; }
  __syncthreads();
  const int w = lane & (ATT_WARPS - 1);
  sum = __reduce_add_sync(FULLM, lane < ATT_WARPS ? red[w] : 0u); longest = __reduce_max_sync(FULLM, red[ATT_WARPS + w]); shortest = __reduce_min_sync(FULLM, red[2 * ATT_WARPS + w]);
  const u32 total = (u32)n_kv * (sum + (u32)(EXTRA * B)), share = (total + ctas - 1) / ctas, most = share + EXTRA;
  f.row = f.kvh = f.at = f.tiles = f.tokens = 0; f.pair = -1;
  if (pairs <= ctas) {
    const u32 lo = max((u32)least, ((u32)n_kv * sum + ctas - 1) / ctas), hi = max(lo, share + SLACK), same = (u32)(ctas / pairs), even = (longest + same - 1) / same;
    f.share = 0;
    if (even <= min(hi, lo + 2 + lo / 16)) {           // rows of about one length, or so few tiles that nothing is left to gain: as many pieces of every pair
      if (warp != 0) return;
      const int pair = cta / (int)same, r = pair / n_kv;
      if (pair < pairs) {
        const int t = tiles_in(held[r]), chunk = (t + (int)same - 1) / (int)same;
        f.at = 1; f.pair = pair; f.split = cta - pair * (int)same; f.ns = (int)same; f.tokens = held[r];
        f.range[0] = min(f.split * chunk, t); f.range[1] = min(chunk, t - f.range[0]);
      }
      return;
    }
    // sixteen sizes between the smallest that might do and share, a warp each (one after the other by bisection they took 0.5 us)
    auto pieces_of = [&](int r, u32 C) { return r < B ? max(1u, ((u32)tiles_in(held[r]) + C - 1) / C) : 0u; };
    {
      const u32 C = lo + ((hi - lo) * (u32)(warp + 1) + ATT_WARPS - 1) / ATT_WARPS;
      u32 n = 0u;
      for (int r = lane; r < B; r += 32) n += pieces_of(r, C);
      n = (u32)n_kv * __reduce_add_sync(FULLM, n);
      if (lane == 0) red[3 * ATT_WARPS + warp] = n <= (u32)ctas ? C : 0xFFFFFFFFu;
    }
    __syncthreads();
    const u32 C = __reduce_min_sync(FULLM, red[3 * ATT_WARPS + w]);
    if (C != 0xFFFFFFFFu) {
      if (warp != 0) return;
      f.at = 1;
      u32 before = 0u;
      for (int r0 = 0; r0 < B; r0 += 32) {
        const u32 n = pieces_of(r0 + lane, C), own = (u32)n_kv * n;
        u32 inc = own;
        scan_step(inc, 1); scan_step(inc, 2); scan_step(inc, 4); scan_step(inc, 8); scan_step(inc, 16);
        const u32 past = __ballot_sync(FULLM, before + inc > (u32)cta);
        if (past) {                                   // the row that the CTA's piece is of
          const int l = __ffs((int)past) - 1, rest = cta - (int)(before + __shfl_sync(FULLM, inc - own, l)), t = tiles_in(held[r0 + l]);
          f.ns = (int)__shfl_sync(FULLM, n, l); f.tokens = held[r0 + l];
          const int h = rest / f.ns, chunk = (t + f.ns - 1) / f.ns;
          f.pair = (r0 + l) * n_kv + h; f.split = rest - h * f.ns;
          f.range[0] = min(f.split * chunk, t); f.range[1] = min(chunk, t - f.range[0]);
          break;
        }
        before += __shfl_sync(FULLM, inc, 31);
      }
      return;
    }
  } else {
    const int k = (pairs + ctas - 1) / ctas;
    if (B <= FLAT_SORT && k <= FLAT_WHOLE && longest <= share && (u32)k * (EXTRA + shortest) <= most && longest < 1u << 22) {
      static_assert(FLAT_SORT <= 512, "nine bits of a key");
      const int mine = tid < B ? tiles_in(held[tid]) << 9 | (511 - tid) : -1;           // (no two alike)
      keys[tid] = mine;
      __syncthreads();
      int rank = 0;
      for (int j = 0; j < B; j += 4) {
        const int4 other = *reinterpret_cast<const int4*>(keys + j);
        rank += (other.x > mine) + (other.y > mine) + (other.z > mine) + (other.w > mine);
      }
      if (tid < B) order[rank] = tid;
      __syncthreads();
      auto place = [&](int i, int c) { return i & 1 ? (i + 1) * ctas - 1 - c : i * ctas + c; };
      u32 load = 0u;
      for (int c = tid; c < ctas; c += ATT_THREADS) {
        u32 own = 0u;
        for (int i = 0; i < k; i++)
          if (place(i, c) < pairs) own += EXTRA + tiles_in(held[order[place(i, c) / n_kv]]);
        load = max(load, own);
      }
      load = __reduce_max_sync(FULLM, load);
      if (lane == 0) red[3 * ATT_WARPS + warp] = load;
      __syncthreads();
      if (__reduce_max_sync(FULLM, red[3 * ATT_WARPS + w]) <= most) {
        if (warp == 0) {
          f.share = -1; f.at = place(k - 1, cta) < pairs ? k : k - 1;
          if (lane < f.at) { const int at = place(lane, cta), r = order[at / n_kv]; window[lane] = r * n_kv + at % n_kv; window[32 + lane] = held[r]; }
          __syncwarp();
        }
        return;
      }
    }
  }
  if (warp != 0) return;
  auto tokens_at = [&](int r) { return r < FLAT_ROWS ? held[r] : tokens_of(r); };
  f.share = (int)share;
  f.lo = (int)min((long)cta * f.share, (long)total); f.hi = (int)min((long)f.lo + f.share, (long)total);
  f.row = B;
  u32 before = 0u;
  for (int r0 = 0; r0 < B && f.lo < f.hi; r0 += 32) {
    const int tokens = r0 + lane < B ? tokens_at(r0 + lane) : 0, t = tiles_in(tokens);
    const u32 own = r0 + lane < B ? (u32)(n_kv * (EXTRA + t)) : 0u;
    u32 inc = own;
    scan_step(inc, 1); scan_step(inc, 2); scan_step(inc, 4); scan_step(inc, 8); scan_step(inc, 16);
    const u32 past = __ballot_sync(FULLM, before + inc > (u32)f.lo);
    if (past) {                                       // the row that the CTA's first place lies in
      const int l = __ffs((int)past) - 1;
      f.row = r0 + l; f.tiles = __shfl_sync(FULLM, t, l);
      const int row_at = (int)(before + __shfl_sync(FULLM, inc - own, l));
      f.kvh = (f.lo - row_at) / (EXTRA + f.tiles);
      f.at = row_at + f.kvh * (EXTRA + f.tiles);
      window[lane] = tokens;
      __syncwarp();
      break;
    }
    before += __shfl_sync(FULLM, inc, 31);
  }
}
// The next piece, by the whole of warp 0.  On the line, window has the tokens of the 32 rows that the walk is among.
template <int EXTRA, class F> __device__ __forceinline__ void flat_next(FlatWalk& f, int B, int n_kv, int lane, int* window, const F& tokens_of) {
  if (f.share <= 0) {
    if (f.at == 0) f.pair = -1;
    else if (--f.at, f.share < 0) { f.pair = window[f.at]; f.tokens = window[32 + f.at]; f.range[0] = 0; f.range[1] = tiles_in(f.tokens); f.split = 0; f.ns = 1; }
    return;
  }
  f.pair = -1;
  while (f.row < B && f.pair < 0) {
    const int first = f.at + EXTRA - (f.tiles > 0 ? 0 : 1), last = first + max(f.tiles, 1) - 1;
    if (first >= f.hi) return;
    if (last >= f.lo) {
      const int c0 = first / f.share;
      f.pair = f.row * n_kv + f.kvh; f.split = blockIdx.x - c0; f.ns = last / f.share - c0 + 1; f.tokens = window[f.row % 32];
      f.range[0] = f.tiles > 0 ? max(f.lo, first) - first : 0; f.range[1] = f.tiles > 0 ? min(f.hi - 1, last) - first + 1 - f.range[0] : 0;
    }
    f.at += EXTRA + f.tiles;
    if (++f.kvh == n_kv) {
      f.kvh = 0;
      if (++f.row < B) {
        if (f.row % 32 == 0) {
          __syncwarp();
          window[lane] = f.row + lane < B ? tokens_of(f.row + lane) : 0;
          __syncwarp();
        }
        f.tiles = tiles_in(window[f.row % 32]);
      }
    }
  }
}

static_assert(FLAT_SCRATCH <= ATT_WARPS * AREA_BYTES, "planned in the segment areas");

// Ranges of a row of a grid, where its length is only known here: the caller goes by a bound on the rows' lengths, the width of a block table or a capacity, and its split count (ns, the most there
// may be) may be far too large for the rows that there are.  A row of up to `one` tiles is not split;  beyond, ranges go down to four tiles until there are 16 of them (24 at head_dim 256, whose CTAs
// work on eight tiles at a time), then down to a tile per warp (`turn`: tiles that a CTA works on at a time).  CTAs that get none leave before they load anything.  So the callers' rules may fill one
// wave: in a table of 2048 tokens 4 x 4 rows of 53 took 9.8 us in nine ranges each, 7.0 by shares of units and take 6.5 now;  in one of 8192 at head_dim 256 a row of 2000 17.5 in 128 ranges, now 10.1.
__device__ __forceinline__ void fewer_ranges(int tiles, int one, int turn, int& ns, int& chunk) {
  if (tiles <= one) { ns = 1; chunk = tiles; return; }
  const int least = max(4, min(turn, turn == ATT_WARPS ? (tiles + 15) >> 4 : tiles / 24));
  if (chunk >= least) return;
  ns = (tiles + least - 1) / least;
  chunk = (tiles + ns - 1) / ns;                     // (as sum_exact takes it)
}
// How the rows are shared out.  GRID: (row, kv head) x splits;  BOUND: the same with fewer_ranges;  TEAM: below;  SHARED: a balanced launch;  FLAT_LINE: above.  Instantiations of their own: the
// shares cost the others registers that the main loop has none of, 1.5 % at 64K tokens, and fewer_ranges costs rows of one to five tiles in several waves, which have one range each, 0.08 us a wave
// (paged 128 x 4 of 30-60 tokens 22.8 -> 22.4, 64 x 8 of 16-80 22.3 -> 21.9, 512 x 8 of 1-80 151 -> 149).
enum { GRID, SHARED, FLAT_LINE, TEAM, BOUND };
// ---- teams: the ranges of a row as one cluster, at most eight CTAs (the portable size), whose partials meet in the shared memory of the first.  Through global memory they take a fence
// until the partials have arrived there, an atomic, and a load of each back, 1.7 us of a launch of 7; through distributed shared memory 0.7: 8 heads x 500 tokens 7.2 -> 6.1 us in a graph.  The others
// store into the first CTA and leave; it has said, ahead of its main loop, that the place is free, which is in the stages that a range of at most TEAM_TILES tiles does not reach and
// that nobody has used before, the queries' way through the last of them included: so the word needs no release, which would take 0.4 us.  Longer ranges, found out
// only here where the caller goes by a bound, take the other way: both decide by the row's length, so the CTAs of a cluster agree.
constexpr int TEAM_MOST = 8, TEAM_STAGE = 6, TEAM_TILES = TEAM_STAGE * TPS;
constexpr int Q_PLACE = TB_RING + NSTG * STAGE_BYTES - 2048;          // where one warp leaves the queries for the others: the end of the last stage
static_assert(TEAM_STAGE * STAGE_BYTES + (TEAM_MOST - 1) * 8 * 130 * 4 <= Q_PLACE - TB_RING && Q_PLACE % 16 == 0, "the partials lie in stages that so few tiles do not reach, ahead of the queries");
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ u32 cluster_address(u32 at, u32 rank) { u32 v; asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(v) : "r"(at), "r"(rank)); return v; }
__device__ __forceinline__ void cluster_store(u32 at, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory"); }

template <bool PAGED, bool DUMP, int NSET, int MODE>
__global__ void __launch_bounds__(ATT_THREADS, 1) decode_attn_kernel(const __grid_constant__ AttnParams p) {
  constexpr bool SHARE = MODE == SHARED, FLAT = MODE == FLAT_LINE, ROWS = MODE == GRID || MODE == TEAM || MODE == BOUND;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_next, s_last, s_split, s_ns, s_tail, s_esc[6];
  __shared__ int s_team;        // (from s_split on: not needed inside the main loop, whose registers are all taken)
  __shared__ FlatWalk s_flat;
  __shared__ int s_rows[FLAT ? 64 : 1];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(FULLM, tid >> 5, 0);   // the same value, but known to the compiler to be uniform across the warp
  const int G = p.G;
  const u32 smem_s = (u32)__cvta_generic_to_shared(smem);
  // ---- programmatic dependent launch: the grid is launched with stream serialisation relaxed, so its CTAs can be made
  // resident while the previous kernel of the stream is still finishing (its split merge runs on a few SMs only).  What does not
  // depend on memory is set up before the wait; nothing is read before that kernel has completed; the next kernel of the stream may be
  // staged behind this one as soon as all of this grid's CTAs are there, whatever they wait for (it waits in turn, and nobody needs the SMs that it takes any more): said ahead of the wait, layers
  // back to back take 6.05 -> 5.8 us at 500 tokens and 47.3 -> 47.0 at 65536.  Both instructions are no-ops in a plain launch.
  if (tid < 256) fill_attn_tables(smem, tid);
  // Warp w fills stage w first, and clears the words of its tiles: a lane that publishes one has cleared it itself, so no other warp has to be waited for.
  auto begin_ring = [&](bool again) {
    if (warp < NSTG && lane < TPS) reinterpret_cast<u32*>(smem + TB_USE)[warp * TPS + lane] = 0u;
    if (lane == 0 && warp < NSTG) {
      if (again) asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_s + TB_FULL + 8 * warp) : "memory");
      mbar_init(smem_s + TB_FULL + 8 * warp, 1);
      reinterpret_cast<int*>(smem + TB_LEFT)[warp] = 0;
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncwarp();
  };
  begin_ring(false);
  // What the grid's own numbering gives is worked out ahead of the wait: the divisions are a quarter of the time from there to the first copy.
  int bh = blockIdx.x, b = bh / p.n_kv, kvh = bh - b * p.n_kv, chunk_all = ROWS && !PAGED ? (((p.S_uniform + 15) >> 4) + p.nsplit - 1) / p.nsplit : 0;
  if (ROWS) asm volatile("" : "+r"(b), "+r"(kvh), "+r"(chunk_all));
  asm volatile("griddepcontrol.launch_dependents;" ::);
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // Which (row, kv head, split) this CTA works on.  Normally the grid says so.  With a row order (ragged paged batches) the CTAs
  // are numbered in the order the hardware hands them out (x fastest) and that number walks the rows from the longest to the
  // shortest, all CTAs of a row together: the big CTAs start first and the small ones fill the SMs at the end.
  int split0 = blockIdx.y, S_paged = 0, ns0 = p.nsplit;
  if (SHARE) {
    int len = 0, row;
    if (lane < p.B) {
      if (PAGED) len = p.seq_len[lane];
      else { const int sl = p.slot[lane]; len = sl < 0 ? 0 : p.seq_len[(long)sl * p.n_kv]; }        // a slot's first head stands for all of its heads
    }
    row_share((len + 15) >> 4, p.B, p.units, p.wave, blockIdx.y, lane, row, split0, ns0);
    if (row >= p.B) return;
    bh = row * p.n_kv + blockIdx.x;
    S_paged = __shfl_sync(FULLM, len, row);
  } else if (PAGED) {
    // the row's token count for the grid's own numbering; the loads of the row order travel at the same time, so a batch whose
    // order is not used pays no extra latency for having one
    S_paged = p.seq_len[b];
    if (p.row_order) {
      const int linear = blockIdx.y * gridDim.x + blockIdx.x, per_row = p.n_kv * p.nsplit;
      const int rr = linear / per_row, rem = linear - rr * per_row;
      const int2 e = p.row_order[rr], use = p.row_order[p.B];
      if (use.x) { bh = e.x * p.n_kv + rem / p.nsplit; split0 = rem % p.nsplit; S_paged = e.y; }
      // the numbers came out of memory: tell the compiler that they are the same in every lane (see below)
      bh = __shfl_sync(FULLM, bh, 0); split0 = __shfl_sync(FULLM, split0, 0);
      b = bh / p.n_kv; kvh = bh - b * p.n_kv;
    }
  }
  auto tokens_of = [&](int row) -> int {              // (a slot's first head stands for all of its heads)
    if (PAGED) return p.seq_len[row];
    const int sl = p.slot[row];
    return sl < 0 ? 0 : p.seq_len[(long)sl * p.n_kv];
  };
  if (FLAT) {
    FlatWalk f;
    flat_plan<FLAT_EXTRA, FLAT_SLACK>(f, p.B, p.n_kv, 4, s_rows, reinterpret_cast<int*>(smem + TB_AREA), tokens_of);
    if (tid == 0) s_flat = f;
    __syncwarp();
  }
  do {
  if (FLAT) {                                        // the next piece
    if (warp == 0) {
      FlatWalk f = s_flat;
      __syncwarp();
      flat_next<FLAT_EXTRA>(f, p.B, p.n_kv, lane, s_rows, tokens_of);
      if (lane == 0) { s_flat = f; s_split = f.split; s_ns = f.ns; }
    }
    __syncthreads();
    bh = __shfl_sync(FULLM, s_flat.pair, 0);
    if (bh < 0) return;
    if (PAGED) S_paged = s_flat.tokens;
  }
  if (!ROWS) { b = bh / p.n_kv; kvh = bh - b * p.n_kv; }

  // ---- which cache head, how many tokens, this CTA's tile range [tlo, tlo + n)
  // (without a slot map row b reads slot b; without a length table every head holds S_uniform tokens: the two dependent
  // loads at the head of the prologue disappear for callers whose heads are all alike, which is what two Pages are)
  int S, ch = 0, TL = 0, ohk = 0, ohv = 0;
  if (PAGED) { S = S_paged; }
  else {
    const int sl = p.slot ? p.slot[b] : b;
    ch = (sl < 0 ? 0 : sl) * p.n_kv + kvh;
    const int s_ld = p.seq_len ? p.seq_len[ch] : p.S_uniform;           // these four loads do not depend on one another
    const int t_ld = p.tail_len ? p.tail_len[ch] : 0;
    ohk = p.K.head_start[ch]; ohv = p.V.head_start[ch];
    S = sl < 0 ? 0 : s_ld;
    TL = sl < 0 ? 0 : t_ld;
  }
  // These values are the same in every thread, but they were loaded from memory: passing them through a shuffle tells the
  // compiler so, and the address arithmetic built on them stays in uniform registers.
  S = __shfl_sync(FULLM, S, 0); ch = __shfl_sync(FULLM, ch, 0); TL = __shfl_sync(FULLM, TL, 0);
  const int ntiles = (S + 15) >> 4;
  int chunk = ROWS && !PAGED && !p.seq_len ? chunk_all : (ntiles + ns0 - 1) / ns0;
  if (MODE == TEAM || MODE == BOUND) {
    if (PAGED || p.seq_len) { fewer_ranges(ntiles, ATT_WARPS, ATT_WARPS, ns0, chunk); if (split0 >= ns0) return; }
    if (tid == 0) s_ns = ns0;
  }
  const int tlo = FLAT ? min(__shfl_sync(FULLM, s_flat.range[0], 0), ntiles) : min(split0 * chunk, ntiles);
  // (the last piece of a pair has what there is to the end, should a head be longer than the first one)
  const int n = FLAT ? (__shfl_sync(FULLM, s_split + 1 - s_ns, 0) == 0 ? ntiles - tlo : min(__shfl_sync(FULLM, s_flat.range[1], 0), ntiles - tlo)) : min(chunk, ntiles - tlo);
  const int nstages = (n + TPS - 1) / TPS;

  auto meta_of = [&](int i) -> TileMeta {             // i counts from the first tile of the CTA's range
    const int tile = tlo + i;
    if (PAGED) { const int pc = p.bt[(long)b * p.bt_stride + tile] * (2 * p.n_kv) + 2 * kvh; return TileMeta{p.mt[pc], p.mt[pc + 1]}; }
    const long at = (long)ch * (p.S_pad >> 4) + tile;
    return TileMeta{p.K.tile_off[at], p.V.tile_off[at]};
  };
  // ---- filling a stage.  What a copy is given comes from uniform values or through a shuffle, so that the compiler knows it to be the same in every lane: the copy
  // instruction takes uniform registers, and anything else costs it a loop over the lanes.
  constexpr int FAR = 1 << 28;                        // "until the end of the allocation", as an escape offset
  auto stage_meta = [&](int st) -> TileMeta {         // lane t < TPS: of tile t;  slot layout, lane TPS: of the tile behind, where the stage's escape bytes end
    const int i = st * TPS + lane;
    if (PAGED) return lane < TPS && i < n ? meta_of(i) : TileMeta{-1, -1};
    return lane <= TPS && (i < n || tlo + i < ntiles) ? meta_of(i) : TileMeta{FAR, FAR};
  };
  // Escape window of a side for tiles whose escape bytes are [m0, m1) of the head's: from the 16-byte boundary at or below the first byte, a
  // multiple of 16 bytes, at most SIDE_ESC, inside the allocation (no bytes when the boundary lies before it).  phase: of the head's first byte;  to_end: bytes from there
  // to the end of the allocation.
  struct HeadEsc { int ohk, ohv, phk, phv, k_end, v_end; };
  auto esc_window = [&](int to_end, int phase, int oh, int m0, int m1, int& start, u32& bytes) {
    const int w16 = (phase + m0) & 15, left = (int)((u32)to_end - (u32)m0 + (u32)w16);
    start = m0 - w16;
    bytes = oh < w16 - m0 || to_end < m0 - w16 ? 0u : (u32)max(0, min(min(SIDE_ESC, (m1 - m0 + w16 + 15) & ~15), left & ~15));
  };
  const u32 slot_bytes = PAGED ? (u32)min(p.TS, PSLOT) : 0u;                   // a paged slot is one contiguous piece, escapes included
  // Both are executed by a whole warp.  The part that needs no metadata (slot layout) ..
  auto fill_payload = [&](int st) {
    const u32 mb = smem_s + TB_FULL + 8 * (st % NSTG), dst = smem_s + TB_RING + (st % NSTG) * STAGE_BYTES, cnt = (u32)min(TPS, n - st * TPS);
    const long row = (long)ch * p.S_pad + (long)(tlo + st * TPS) * T;
    warp_add_tx(mb, 2 * cnt * (TILE_SM + TILE_CD + 4 * T));
    warp_g2s(dst + SB_FL, reinterpret_cast<const uint8_t*>(p.K.flags) + row * 4, cnt * 4 * T, mb);
    warp_g2s(dst + SIDE_BYTES + SB_FL, reinterpret_cast<const uint8_t*>(p.V.flags) + row * 4, cnt * 4 * T, mb);
    warp_g2s(dst, p.K.sm + row * D, cnt * TILE_SM, mb); warp_g2s(dst + SB_CD, p.K.codes + row * CB, cnt * TILE_CD, mb);
    warp_g2s(dst + SIDE_BYTES, p.V.sm + row * D, cnt * TILE_SM, mb); warp_g2s(dst + SIDE_BYTES + SB_CD, p.V.codes + row * CB, cnt * TILE_CD, mb);
  };
  // .. and the rest, or all of a paged stage.  own: stage_meta
  auto fill_rest = [&](int st, const TileMeta& own, const HeadEsc& h) {
    const int slot = st % NSTG;
    const u32 mb = smem_s + TB_FULL + 8 * slot, dst = smem_s + TB_RING + slot * STAGE_BYTES;
    int4 info;
    u32 pieces = 0u;
    int k0 = 0, v0 = 0; u32 nk = 0u, nv = 0u;
    if (PAGED) {
      const u32 e = dst + 2 * lane * PSLOT + SLOT_OVF_OFF;
      const int avail = min(p.ovf_slot, (int)slot_bytes - SLOT_OVF_OFF);
      info = make_int4((int)e, avail, (int)(e + PSLOT), avail);
      pieces = (u32)popc(__ballot_sync(FULLM, own.mk >= 0)) + (u32)popc(__ballot_sync(FULLM, own.mv >= 0));
    } else {
      const int m0k = __shfl_sync(FULLM, own.mk, 0), m0v = __shfl_sync(FULLM, own.mv, 0), m1k = __shfl_sync(FULLM, own.mk, TPS), m1v = __shfl_sync(FULLM, own.mv, TPS);
      esc_window(h.k_end, h.phk, h.ohk, m0k, m1k, k0, nk); esc_window(h.v_end, h.phv, h.ohv, m0v, m1v, v0, nv);
      info = make_int4((int)dst + SB_ESC + own.mk - k0, (int)nk - (own.mk - k0), (int)dst + SIDE_BYTES + SB_ESC + own.mv - v0, (int)nv - (own.mv - v0));
    }
    if (lane < min(TPS, n - st * TPS)) {
      reinterpret_cast<int4*>(smem + TB_ESC)[slot * TPS + lane] = info;
      reinterpret_cast<int2*>(smem + TB_META)[slot * TPS + lane] = make_int2(own.mk, own.mv);
      asm volatile("st.relaxed.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_s + TB_USE + 4 * (slot * TPS + lane)), "r"((u32)(st + 1) << 4 | (PAGED && own.mk < 0 ? 4u : 0u) | (PAGED && own.mv < 0 ? 8u : 0u)) : "memory");
    }
    __syncwarp();
    warp_expect_tx(mb, PAGED ? pieces * slot_bytes : nk + nv);
    if (PAGED) {
#pragma unroll
      for (int t = 0; t < TPS; t++) {
        const int k = __shfl_sync(FULLM, own.mk, t), v = __shfl_sync(FULLM, own.mv, t);
        if (k >= 0) warp_g2s(dst + 2 * t * PSLOT, p.buf + (long)k * p.TS, slot_bytes, mb);
        if (v >= 0) warp_g2s(dst + (2 * t + 1) * PSLOT, p.buf + (long)v * p.TS, slot_bytes, mb);
      }
    } else {
      if (nk > 0) warp_g2s(dst + SB_ESC, p.K.ovf + ((long)h.ohk + k0), nk, mb);
      if (nv > 0) warp_g2s(dst + SIDE_BYTES + SB_ESC, p.V.ovf + ((long)h.ohv + v0), nv, mb);
    }
  };

  // ---- prologue.  HBM is idle when the grid starts and every CTA asks at once: what the first tiles need goes first, the small loads ahead of the first stages' payload (which needs
  // no metadata in the slot layout), the other stages when the first tiles are there.  Each kind of load has warps of its own, since a warp comes to the barrier when its last
  // load is back: bases, queries, metadata and payload.  us from the end of the grid's wait to the first tile, 8 heads x 500 tokens 2.5 -> 1.7, x 65536 3.7 -> 3.5 (there the first
  // stages of all CTAs are 14 MB).
  constexpr int FIRST = (ATT_WARPS + TPS - 1) / TPS;
  const bool filler = warp < min(NSTG, nstages);                               // warp w fills stage w
  TileMeta ahead{};
  // The queries, by one warp for all, through the last stage's place, which is not filled before the second barrier.  Every warp on its own asked for them behind the first stages'
  // payload and had them 1.1 us later.  (Not in a flat launch, whose pieces begin at different times: 425 -> 433 us for 16 x 4096..65536.)
  static_assert(FIRST < NSTG && 2048 <= STAGE_BYTES, "the last stage is not one of the first");
  uint4* const q_place = reinterpret_cast<uint4*>(smem + Q_PLACE) + lane;
  QFrag Q;
  if (!FLAT && warp == ATT_WARPS - 3) {
    load_q(Q, p.q + ((long)b * p.n_q + kvh * G) * D, D, G, lane);
#pragma unroll
    for (int i = 0; i < 4; i++) q_place[32 * i] = make_uint4(Q.qa[2 * i][0], Q.qa[2 * i][1], Q.qa[2 * i + 1][0], Q.qa[2 * i + 1][1]);
  }
  if (filler) {
    ahead = stage_meta(warp);
    if (!PAGED && warp < FIRST) fill_payload(warp);
  }
  if (FLAT) load_q(Q, p.q + ((long)b * p.n_q + kvh * G) * D, D, G, lane);
  ohk = __shfl_sync(FULLM, ohk, 0); ohv = __shfl_sync(FULLM, ohv, 0);          // (not before: whoever needs them waits for them)
  const HeadEsc head_esc{ohk, ohv, PAGED ? 0 : (int)((reinterpret_cast<uintptr_t>(p.K.ovf) + (unsigned)ohk) & 15), PAGED ? 0 : (int)((reinterpret_cast<uintptr_t>(p.V.ovf) + (unsigned)ohv) & 15),
                         PAGED ? 0 : (int)max(-1L, min((long)p.K.ovf_bytes - ohk, 0x7FFFFF00L)), PAGED ? 0 : (int)max(-1L, min((long)p.V.ovf_bytes - ohv, 0x7FFFFF00L))};
  {
    const int brow = PAGED || p.n_base_rows == p.n_kv ? kvh : ch < p.n_base_rows ? ch : ch % p.n_base_rows;
    if (warp == ATT_WARPS - 2 && lane < 16) fill_pair_bases<false>(smem + TB_BASES, (PAGED ? p.b3k : p.K.base3) + brow * D, (PAGED ? p.b4k : p.K.base4) + brow * D, lane);
    if (warp == ATT_WARPS - 1 && lane < 16) fill_pair_bases<true>(smem + TB_BASES, (PAGED ? p.b3v : p.V.base3) + brow * D, (PAGED ? p.b4v : p.V.base4) + brow * D, lane);
    if (SHARE && tid == 0) s_split = split0;
    if (SHARE && tid == 0) s_ns = ns0;
    if (FLAT && tid == 0) s_tail = TL;
    if (tid == 0) s_next = ATT_WARPS;                        // tiles 0 .. W-1 of the range go to warps 0 .. W-1, the rest is handed out on demand
  }
  if (filler && warp < FIRST) fill_rest(warp, ahead, head_esc);
  if (!PAGED && tid == 0) *reinterpret_cast<HeadEsc*>(s_esc) = head_esc;
  WarpAcc<NSET> A;
  A.clear();
  __syncthreads();
  if (!FLAT) {
#pragma unroll
    for (int i = 0; i < 4; i++) { const uint4 w = q_place[32 * i]; Q.qa[2 * i][0] = w.x; Q.qa[2 * i][1] = w.y; Q.qa[2 * i + 1][0] = w.z; Q.qa[2 * i + 1][1] = w.w; }
    __syncthreads();
  }
  if (MODE == TEAM) {
    const bool team = ns0 > 1 && chunk <= TEAM_TILES;
    if (tid == 0) s_team = team;
    __syncwarp();
    if (team) cluster_arrive();                      // (the places of the partials are free)
  }
  if (filler && warp >= FIRST) {                     // (where all CTAs begin together, behind the warp's own first tile: any earlier, and these copies hold back the first stages')
    u32 flags;
    if (!FLAT) __all_sync(FULLM, mbar_wait_use(smem_s + TB_FULL + 8 * (warp / TPS), 0u, smem_s + TB_USE + 4 * warp, (u32)(warp / TPS) + 1u, flags));          // (one that runs out is met again in the main loop)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");               // the queries came through the last stage by ordinary stores
    if (!PAGED) fill_payload(warp);
    fill_rest(warp, ahead, head_esc);
  }

  uint16_t* const dump_k = DUMP ? p.dump_k + (long)bh * p.dump_S * D : nullptr;
  uint16_t* const dump_v = DUMP ? p.dump_v + (long)bh * p.dump_S * D : nullptr;
  const AttnView W = attn_view(smem_s, smem_s + TB_BASES);
  // ---- main loop.  The warp's first tile is tile `warp` of the range; every further one is taken from the CTA's counter at the top of the
  // iteration, one tile ahead of its use, so fast and slow warps finish within about one tile of each other.  The warp that is the
  // last to leave a stage fills it again with the tiles NSTG stages on.
  const u32 area = smem_s + TB_AREA + warp * AREA_BYTES, next_at = (u32)__cvta_generic_to_shared(&s_next);
  int it = warp;
  while (it < n) {
    int nx = lane_inc<false>(next_at, lane);
    const int st = it / TPS, ti = it % TPS, slot = st % NSTG, tile = tlo + it, nth = it % (TPS * NSTG);
    u32 flags;
    if (!__all_sync(FULLM, mbar_wait_use(smem_s + TB_FULL + 8 * slot, (u32)(st / NSTG) & 1u, smem_s + TB_USE + 4 * nth, (u32)st + 1u, flags))) {     // the whole warp gives up together
      if (lane == 0) atomicExch(p.err, 1);
      break;
    }
    const int nvalid = min(T, S - tile * T);
    const bool rawk = PAGED && (flags & 4u), rawv = PAGED && (flags & 8u);
    const int2 own = reinterpret_cast<const int2*>(smem + TB_ESC)[2 * nth + (lane >> 4)];           // the lane's side: where its escape bytes are
    const u32 stage = smem_s + TB_RING + slot * STAGE_BYTES;
    const u32 fl = PAGED ? stage + (2 * ti + (lane >> 4)) * PSLOT + SLOT_FL_OFF : stage + (lane >> 4) * SIDE_BYTES + SB_FL + 4 * T * ti;
    const int win = plan_tile(!(lane >> 4 ? rawv : rawk), fl, (u32)own.x, own.y, W, area, PATCH_MAX, lane);
    const int2 m = reinterpret_cast<const int2*>(smem + TB_META)[nth];
    const uint8_t* const s0 = smem + TB_RING + slot * STAGE_BYTES;
    const SideView ks = PAGED ? SideView{s0 + 2 * ti * PSLOT, s0 + 2 * ti * PSLOT + SLOT_CD_OFF, p.buf + (long)m.x * p.TS + SLOT_OVF_OFF}
                              : SideView{s0 + ti * TILE_SM, s0 + SB_CD + ti * TILE_CD, p.K.ovf + ((long)s_esc[0] + m.x)};
    const SideView vs = PAGED ? SideView{s0 + (2 * ti + 1) * PSLOT, s0 + (2 * ti + 1) * PSLOT + SLOT_CD_OFF, p.buf + (long)m.y * p.TS + SLOT_OVF_OFF}
                              : SideView{s0 + SIDE_BYTES + ti * TILE_SM, s0 + SIDE_BYTES + SB_CD + ti * TILE_CD, p.V.ovf + ((long)s_esc[1] + m.y)};
    float sc[4] = {0.f, 0.f, 0.f, 0.f};
    if (!rawk) k_tile<DUMP>(sc, ks, win, area, W, lane, Q, dump_k + (long)tile * T * D, nvalid);
    else raw_scores<DUMP>(sc, p.raw + (long)raw_tile(m.x) * (T * D), nvalid, lane, Q, dump_k + (long)tile * T * D);
    nx = __shfl_sync(FULLM, nx, 0);
    const bool asks = ti == TPS - 1 && st + NSTG < nstages;
    if (asks) ahead = stage_meta(st + NSTG);                                 // for the warp that will fill the stage again
    PFrag<NSET> P;
    if (nvalid == T) softmax_step<NSET, true>(A, sc, p.scale_log2, nvalid, lane, P);
    else softmax_step<NSET, false>(A, sc, p.scale_log2, nvalid, lane, P);
    if (!rawv) v_tile<DUMP, NSET>(A, vs, win, area, W, lane, P, dump_v + (long)tile * T * D, nvalid);
    else raw_accum<DUMP, NSET>(A, p.raw + (long)raw_tile(m.y) * (T * D), nvalid, lane, P, dump_v + (long)tile * T * D);
    if (asks && lane <= TPS) reinterpret_cast<int2*>(smem + TB_NEXT)[slot * (TPS + 1) + lane] = make_int2(ahead.mk, ahead.mv);
    __syncwarp();                                    // every lane is done with the tile and with the area
    if (st + NSTG < nstages) {
      const int left = __shfl_sync(FULLM, lane_inc<true>(smem_s + TB_LEFT + 4 * slot, lane), 0);
      if ((left & (TPS - 1)) == TPS - 1) {
        __syncwarp();
        if (!PAGED) fill_payload(st + NSTG);
        ahead = TileMeta{-1, -1};
        if (lane <= TPS) { const int2 e = reinterpret_cast<const int2*>(smem + TB_NEXT)[slot * (TPS + 1) + lane]; ahead = TileMeta{e.x, e.y}; }
        fill_rest(st + NSTG, ahead, PAGED ? head_esc : HeadEsc{__shfl_sync(FULLM, s_esc[0], 0), __shfl_sync(FULLM, s_esc[1], 0), __shfl_sync(FULLM, s_esc[2], 0), __shfl_sync(FULLM, s_esc[3], 0), __shfl_sync(FULLM, s_esc[4], 0), __shfl_sync(FULLM, s_esc[5], 0)});
      }
    }
    it = nx;
  }
  const int split = SHARE || FLAT ? s_split : split0, NS = MODE == GRID ? p.nsplit : s_ns;
  if (FLAT) { bh = __shfl_sync(FULLM, s_flat.pair, 0); b = bh / p.n_kv; kvh = bh % p.n_kv; TL = __shfl_sync(FULLM, s_tail, 0); }
  // ---- slot layout: the raw BF16 tail belongs to the last split's last warp
  if (!PAGED && TL > 0 && split == NS - 1 && warp == ATT_WARPS - 1) {
    const uint16_t* kraw = reinterpret_cast<const uint16_t*>(p.K.tail) + (long)ch * p.tail_cap * D;
    const uint16_t* vraw = reinterpret_cast<const uint16_t*>(p.V.tail) + (long)ch * p.tail_cap * D;
    for (int t0 = 0; t0 < TL; t0 += T) {
      const int nvalid = min(T, TL - t0);
      float sc[4] = {0.f, 0.f, 0.f, 0.f};
      raw_scores<DUMP>(sc, kraw, nvalid, lane, Q, dump_k + ((long)S + t0) * D);
      PFrag<NSET> P;
      softmax_step<NSET, false>(A, sc, p.scale_log2, nvalid, lane, P);
      raw_accum<DUMP, NSET>(A, vraw, nvalid, lane, P, dump_v + ((long)S + t0) * D);
      kraw += T * D; vraw += T * D;
    }
  }

  // ---- merge the warps of the CTA (the ring is free now)
  if (__syncthreads_or(sum_warp(A))) sum_exact<PAGED, false>(p, smem + TB_RING, bh, split, NS, FLAT ? s_flat.range : nullptr);
  else stage_warp(A, smem + TB_RING, G, warp, lane);
  __syncthreads();
  const long qh0 = (long)b * p.n_q + kvh * G;
  const int d = tid & 127;
  // where a query head's merged (M, L, acc) goes when this is the last word of this GPU on it
  const int x_ep = p.x_recv ? __ldcg(p.x_epoch) : 0;             // number of this exchange - 1; advanced only after every group has read it
  auto deliver = [&](int g, float M, float L, float Ac) {
    const long qh = qh0 + g;
    if (p.x_recv) {                                  // the partial, pushed to every rank's receive buffer over NVLink
      const long row = ((long)((x_ep & 1) * p.x_world + p.x_rank) * p.x_rows_cap + qh) * 130;
      for (int rk = 0; rk < p.x_world; rk++) {
        unsigned long long* o = p.x_recv[rk] + row;
        if (d == 0) { x_store(o, M * LN2, (u32)x_ep + 1u); x_store(o + 1, L, (u32)x_ep + 1u); }
        x_store(o + 2 + d, Ac, (u32)x_ep + 1u);
      }
    } else if (p.part) {                             // un-normalised partial for a cross-GPU merge: m in natural-log units
      float* o = p.part + qh * 130;
      if (d == 0) { o[0] = M * LN2; o[1] = L; }
      o[2 + d] = Ac;
    } else {
      const float v = L > 0.f ? Ac / L : 0.f;
      p.out[qh * D + d] = __bfloat16_as_ushort(__float2bfloat16(v));
      if (p.out_f32) p.out_f32[qh * D + d] = v;
    }
  };
  float M[NSET], Lc[NSET], Ac[NSET];                  // of heads tid / 128 and 4 above
#pragma unroll
  for (int i = 0; i < NSET; i++) {
    const int g = (tid >> 7) + 4 * i;
    if (g >= G) continue;
    merge_warps<ATT_WARPS>(smem + TB_RING, 1, 0, g, d, M[i], Lc[i], Ac[i]);
    if (MODE == TEAM && s_team) continue;
    if (FLAT && NS == 1) deliver(g, M[i], Lc[i], Ac[i]);
    if (NS > 1) {
      const long pidx = FLAT ? (long)(blockIdx.x + bh) * G + g : SHARE ? ((long)blockIdx.x * p.units + blockIdx.y) * G + g : (qh0 + g) * p.nsplit + split;
      if (d == 0) { p.pm[pidx] = M[i]; p.pl[pidx] = Lc[i]; }
      p.pa[pidx * D + d] = Ac[i];
    }
  }
  if (MODE == TEAM && s_team) {
    const float* const parts = reinterpret_cast<const float*>(smem + TB_RING + TEAM_STAGE * STAGE_BYTES);           // [split - 1][8][m, l, acc]
    cluster_wait();
    if (split) {
      const u32 first = cluster_address(smem_s + TB_RING + TEAM_STAGE * STAGE_BYTES, 0u) + (u32)(split - 1) * (8 * 130 * 4);
#pragma unroll
      for (int i = 0; i < NSET; i++) {
        const int g = (tid >> 7) + 4 * i;
        if (g >= G) continue;
        const u32 at = first + (u32)g * (130 * 4);
        if (d == 0) { cluster_store(at, M[i]); cluster_store(at + 4, Lc[i]); }
        cluster_store(at + 8 + 4 * d, Ac[i]);
      }
      __syncwarp();
      cluster_arrive_release();
      return;
    }
    cluster_arrive_release();
    cluster_wait();
#pragma unroll
    for (int i = 0; i < NSET; i++) {
      const int g = (tid >> 7) + 4 * i;
      if (g >= G) continue;
      float m[7], most = M[i];
#pragma unroll
      for (int s = 0; s < 7; s++) { m[s] = s + 1 < NS ? parts[(s * 8 + g) * 130] : -CUDART_INF_F; most = fmaxf(most, m[s]); }
      const float keep = M[i] == -CUDART_INF_F ? 0.f : fast_exp2(M[i] - most);
      float L = Lc[i] * keep, A2 = Ac[i] * keep;
#pragma unroll
      for (int s = 0; s < 7; s++)
        if (s + 1 < NS && m[s] != -CUDART_INF_F) {
          const float f = fast_exp2(m[s] - most);
          L += parts[(s * 8 + g) * 130 + 1] * f; A2 += parts[(s * 8 + g) * 130 + 2 + d] * f;
        }
      deliver(g, most, L, A2);
    }
    return;
  }
  const bool last = NS == 1 || last_split(p.counters + bh, NS, &s_last);        // (of one split there is nothing to merge)
  if (!FLAT && !last) return;
  if (FLAT) { if (NS > 1 && last) merge_pieces<4 * NSET>(p, smem + TB_RING, (long)(blockIdx.x - split + bh) * G, 1, G, G, NS, deliver); }
  else {
#pragma unroll
    for (int i = 0; i < NSET; i++) {
      const int g = (tid >> 7) + 4 * i;
      if (g >= G) continue;
      if (NS > 1) merge_splits<32>(p, SHARE ? ((long)blockIdx.x * p.units + blockIdx.y - split) * G + g : (qh0 + g) * p.nsplit, SHARE ? G : 1, NS, d, M[i], Lc[i], Ac[i]);
      deliver(g, M[i], Lc[i], Ac[i]);
    }
  }
  if (p.x_recv) {
    // Every entry carries the exchange number, so nothing else announces the rows (see x_store / x_load).
    if (!p.x_fused) return;                          // the wait-and-merge runs as its own launch (gaac_exchange_merge)
    // ---- fused: wait (bounded) for the rows of this group from every rank, merge them, write the output
    const unsigned long long* base = p.x_recv[p.x_rank] + (long)(x_ep & 1) * p.x_world * p.x_rows_cap * 130;
    float v[2] = {0.f, 0.f};
    int bad = 0;
    for (int g = tid >> 7, i = 0; g < G; g += ATT_THREADS / 128, i++)
      bad |= !x_merge_rows(base, p.x_world, p.x_rows_cap, qh0 + g, d, (u32)x_ep + 1u, v[i]);
    const int any_bad = __syncthreads_or(bad);       // a group whose rows did not all arrive is reported and comes back as zeros
    if (any_bad && tid == 0) atomicExch(p.x_err, 1);
    for (int g = tid >> 7, i = 0; g < G; g += ATT_THREADS / 128, i++) {
      const long qh = qh0 + g;
      const float o = any_bad ? 0.f : v[i];
      if (p.out) p.out[qh * D + d] = __bfloat16_as_ushort(__float2bfloat16(o));
      if (p.out_f32) p.out_f32[qh * D + d] = o;
    }
    // the exchange number advances when every group of this launch is through (each has read it by then)
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(p.x_ticket, 1) == (int)gridDim.x - 1) { *p.x_ticket = 0; __threadfence(); atomicAdd(p.x_epoch, 1); }
    }
  }
  if (FLAT) {                                        // every copy of the piece has landed, and its last waits are behind this barrier.  (At the top of the loop the same
    __syncthreads();                                 // takes 0.5 us of a short launch and spills.)
    begin_ring(true);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");               // the ring was written by the merges
  }
  } while (FLAT);
}

// ------------------------------------------------------------------------------------------------ head_dim 256, paged layout
// A 256-dim head is stored as two 128-dim half-heads in neighbouring tile slots, each with its own bases
// (gaac/vllm/paged_kernel256.py:1-4): block = 2*n_kv half-heads x {K, V}, half-head hh = 2*kvh + half.  Two warps form a pair that
// streams the same tiles: each warp owns one half - it stages and rebuilds its half's K tile, which yields a partial score, and
// its half's V tile, which yields its 128 output dimensions.  The two partial scores meet in shared memory once per tile (one
// 64-thread named barrier is enough: a warp leaves its scores in its stage, over the K tile that it is done with, which is filled
// again only behind the next tile's barrier), after which both warps run the same softmax step on the same numbers.  Tiles are
// handed to PAIRS from the CTA's counter; the even warp takes the number and passes it on through shared memory.  A warp whose
// bounded wait on its copies runs out says so in the same place, so that both warps of the pair leave the loop together and
// nobody is left at the barrier.
// Output: partials of "virtual heads" vq = 2 * query head + half, which the last CTA of a (row, kv head) merges into out [B, n_q, 256].

// (what shared memory has room for)
constexpr int META256_TILES = 48, PATCH256 = 56, SEG256_BYTES = SEG_PATCH + 8 * PATCH256;
constexpr int CTL_BYTES = 16;                                      // of a pair and tile parity: {next tile, fail flag of half 0, of half 1, -}
constexpr int T256_BASES = ADDEND_BYTES + SEGTAB_BYTES, T256_META = T256_BASES + 2 * PAIR_BASES_BYTES, T256_CTL = T256_META + META256_TILES * 16;
constexpr int T256_SEG = T256_CTL + (ATT_WARPS / 2) * 2 * CTL_BYTES, T256_RING = T256_SEG + ATT_WARPS * SEG256_BYTES;
constexpr int STAGE256_BYTES = 16 + 2 * PSLOT, WARP256_BYTES = 2 * STAGE256_BYTES;      // stage: mbarrier, then the warp's K slot and V slot
constexpr int ATT256_SMEM = T256_RING + ATT_WARPS * WARP256_BYTES + 16;          // (an escape segment is read as whole words)
static_assert(T256_BASES % 16 == 0 && T256_RING % 16 == 0 && T256_META % 16 == 0 && T256_CTL % 16 == 0 && ATT256_SMEM + 336 <= 232448, "one CTA per SM");

static_assert(FLAT_SCRATCH <= ATT_WARPS * SEG256_BYTES, "planned in the segment areas");
// FLAT: see FlatWalk; 8 rows x 4 kv heads of 1K-8K tokens 33.1 -> 24.8 us (22.5 now), 20 x 8 of up to 3K 95 -> 73 (a grid, rows as they come; 63 now).  Pieces of two tiles on short rows: of four
// 0.5 us slower on 2 x 4 of 700.
template <int NSET, bool FLAT>
__global__ void __launch_bounds__(ATT_THREADS, 1) paged256_attn_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_next, s_last, s_ns;
  __shared__ FlatWalk s_flat;
  __shared__ int s_rows[FLAT ? 64 : 1];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(FULLM, tid >> 5, 0);
  const int hf = warp & 1, pair = warp >> 1;
  const int G = p.G, NT = 4 * p.n_kv;                // p.n_kv = 256-dim kv heads; NT tile slots per block
  const int ring = T256_RING + warp * WARP256_BYTES;
  const u32 smem_s = (u32)__cvta_generic_to_shared(smem), ring_s = smem_s + ring;
  if (tid < 256) fill_attn_tables(smem, tid);
  auto begin_ring = [&] {
    if (tid < (ATT_WARPS / 2) * 2 * CTL_BYTES / 4) reinterpret_cast<u32*>(smem + T256_CTL)[tid] = 0u;
    if (lane == 0) {
      mbar_init(ring_s, 1); mbar_init(ring_s + STAGE256_BYTES, 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
  };
  if (!FLAT) begin_ring();
  asm volatile("griddepcontrol.launch_dependents;" ::);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  auto tokens_of = [&](int row) -> int { return p.seq_len[row]; };
  if (FLAT) {
    FlatWalk f;
    flat_plan<FLAT_EXTRA256, FLAT_SLACK256>(f, p.B, p.n_kv, 2, s_rows, reinterpret_cast<int*>(smem + T256_SEG), tokens_of);
    if (tid == 0) s_flat = f;
    __syncwarp();
  }
  int bh = blockIdx.x, split = blockIdx.y, NS = p.nsplit;
  do {
  if (FLAT) {                                        // the next piece
    if (warp == 0) {
      FlatWalk f = s_flat;
      __syncwarp();
      flat_next<FLAT_EXTRA256>(f, p.B, p.n_kv, lane, s_rows, tokens_of);
      if (lane == 0) s_flat = f;
    }
    begin_ring();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");               // the ring was written by the merges of the piece before
    __syncthreads();
    bh = __shfl_sync(FULLM, s_flat.pair, 0); split = __shfl_sync(FULLM, s_flat.split, 0); NS = __shfl_sync(FULLM, s_flat.ns, 0);
    if (bh < 0) return;
  }
  int b = bh / p.n_kv, kvh = bh % p.n_kv;
  // The loads that need no length, queries and bases, beside the first that are waited for: in a grid the length, in a flat launch, which has planned with it, the block table.  Then the table for the
  // pair's first tile and for the tiles whose metadata is kept together, then both of their mode-table entries, so that the barrier waits for three loads behind one another.  (The first tile's chain, then
  // queries, bases and the kept tiles' chain: five to six.)  us, with the return behind the merges: 8 x 4 rows of 1K-8K tokens 23.3 -> 22.5, 9 x 4 of 500-12000 41.7 -> 39.9, 6 x 2 of 4K-60K 66.1 ->
  // 64.1, in a grid 8 x 4 of 510 11.2 -> 10.9.  The second tile of every pair asked for as soon as the first is there: 16.6 -> 16.2 where a pair has two or three, but its branch in the main loop
  // costs a per cent where it has more.
  const int tokens = FLAT ? s_flat.tokens : p.seq_len[b];
  QFrag Q;
  auto load_tables = [&] {
    load_q(Q, p.q + ((long)b * p.n_q + kvh * G) * (2 * D) + hf * D, 2 * D, G, lane);
    if (warp >= 8 && warp < 12) {
      const int h2 = warp & 1, row = (2 * kvh + h2) * D;
      uint8_t* o = smem + T256_BASES + h2 * PAIR_BASES_BYTES;
      if (lane < 16) { if (warp < 10) fill_pair_bases<false>(o, p.b3k + row, p.b4k + row, lane); else fill_pair_bases<true>(o, p.b3v + row, p.b4v + row, lane); }
    }
  };
  if (!FLAT) load_tables();
  const int S = __shfl_sync(FULLM, tokens, 0);
  const int ntiles = (S + 15) >> 4;
  int chunk = (ntiles + NS - 1) / NS;
  if (!FLAT) {
    // (the merge of groups of 5 to 8 is dearer: rows of 9 or 10 tiles, of a table of 36 or 40, 10.6 us in one CTA, 12.3 in ranges of four tiles;  two ranges pay from 24 tiles on)
    if (p.nsplit > 1) fewer_ranges(ntiles, NSET == 1 ? ATT_WARPS / 2 : p.nsplit == 2 ? 24 : 16, ATT_WARPS / 2, NS, chunk);
    if (split >= NS) return;
    if (tid == 0) s_ns = NS;
  }
  const int tlo = min(FLAT ? __shfl_sync(FULLM, s_flat.range[0], 0) : split * chunk, ntiles), n = min(FLAT ? __shfl_sync(FULLM, s_flat.range[1], 0) : chunk, ntiles - tlo);
  int* const ctl_pair = reinterpret_cast<int*>(smem + T256_CTL + pair * (2 * CTL_BYTES));
  const int4* meta_s = reinterpret_cast<const int4*>(smem + T256_META);        // per tile: mode-table entries of {K, V} of half 0, of half 1
  auto slot_of = [&](int i) { return p.bt[(long)b * p.bt_stride + tlo + i] * NT + 4 * kvh; };
  auto meta_of = [&](int i) -> TileMeta {
    if (i < META256_TILES) { const int2 m = reinterpret_cast<const int2*>(meta_s + i)[hf]; return TileMeta{m.x, m.y}; }
    const int pc = slot_of(i) + 2 * hf;
    return TileMeta{p.mt[pc], p.mt[pc + 1]};
  };
  const u32 slot_bytes = (u32)min(p.TS, PSLOT);
  auto issue = [&](u32 st, const TileMeta& m) {                                // executed by lane 0
    // the stage may have been written through ordinary stores (patch numbers): order those before the copy engine's writes
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(st, (m.mk >= 0 ? slot_bytes : 0u) + (m.mv >= 0 ? slot_bytes : 0u));
    if (m.mk >= 0) bulk_g2s(st + 16, p.buf + (long)m.mk * p.TS, slot_bytes, st);
    if (m.mv >= 0) bulk_g2s(st + 16 + PSLOT, p.buf + (long)m.mv * p.TS, slot_bytes, st);
  };
  int it = pair;
  TileMeta cur{0, 0};
  const bool first = it < n, keeps = tid < min(n, META256_TILES);
  const int pc = first ? slot_of(it) + 2 * hf : 0, pk = keeps ? slot_of(tid) : 0;
  if (FLAT) load_tables();
  int4 kept{0, 0, 0, 0};
  if (first) cur = TileMeta{p.mt[pc], p.mt[pc + 1]};
  if (keeps) kept = make_int4(p.mt[pk], p.mt[pk + 1], p.mt[pk + 2], p.mt[pk + 3]);
  if (first && lane == 0) issue(ring_s, cur);
  if (keeps) reinterpret_cast<int4*>(smem + T256_META)[tid] = kept;
  if (tid == 0) s_next = ATT_WARPS / 2;               // tiles 0 .. pairs - 1 of the range go to the pairs in order, the rest is handed out on demand
  WarpAcc<NSET> A;
  A.clear();
  __syncthreads();

  const AttnView W = attn_view(smem_s, smem_s + T256_BASES + hf * PAIR_BASES_BYTES);
  const u32 area = smem_s + T256_SEG + warp * SEG256_BYTES, next_at = (u32)__cvta_generic_to_shared(&s_next);
  int stg = 0, par = 0;
  u32 phase = 0;
  const int avail = min(p.ovf_slot, (int)slot_bytes - SLOT_OVF_OFF);
  while (it < n) {
    int t1 = hf == 0 ? lane_inc<false>(next_at, lane) : 0;
    const bool ok = __all_sync(FULLM, mbar_wait(ring_s + stg * STAGE256_BYTES, (phase >> stg) & 1u));
    phase ^= 1u << stg;
    const int so = ring + stg * STAGE256_BYTES + 16;
    const uint8_t* stage = smem + so;
    const int nvalid = min(T, S - (tlo + it) * T);
    float sc[4] = {0.f, 0.f, 0.f, 0.f};
    const SideView ks{stage, stage + SLOT_CD_OFF, p.buf + (long)cur.mk * p.TS + SLOT_OVF_OFF};
    const SideView vs{stage + PSLOT, stage + PSLOT + SLOT_CD_OFF, p.buf + (long)cur.mv * p.TS + SLOT_OVF_OFF};
    int win = 0;
    if (ok) {
      const u32 t0 = smem_s + so + (lane >> 4) * PSLOT;
      win = plan_tile((lane >> 4 ? cur.mv : cur.mk) >= 0, t0 + SLOT_FL_OFF, t0 + SLOT_OVF_OFF, avail, W, area, PATCH256, lane);
      if (cur.mk >= 0) k_tile<false>(sc, ks, win, area, W, lane, Q, nullptr, nvalid);
      else raw_scores<false>(sc, p.raw + (long)raw_tile(cur.mk) * (T * D), nvalid, lane, Q, nullptr);
    }
    // ---- the two halves' partial scores meet; the next tile's number and a failed wait travel with them
    __syncwarp();                                      // every lane is done with the K tile
    reinterpret_cast<float4*>(smem + so)[lane] = make_float4(sc[0], sc[1], sc[2], sc[3]);
    int* ctl = ctl_pair + par * (CTL_BYTES / 4);
    if (lane == 0) { if (hf == 0) ctl[0] = t1; if (!ok) ctl[1 + hf] = 1; }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
    const float4 other = reinterpret_cast<const float4*>(smem + so + (hf ? -WARP256_BYTES : WARP256_BYTES))[lane];      // the same stage of the other warp
    sc[0] += other.x; sc[1] += other.y; sc[2] += other.z; sc[3] += other.w;
    t1 = ctl[0];
    const bool failed = (ctl[1] | ctl[2]) != 0;
    par ^= 1;
    if (failed) { if (lane == 0) atomicExch(p.err, 1); break; }                 // both warps of the pair see the same flags and leave together
    TileMeta nxt{0, 0};
    if (t1 < n) { nxt = meta_of(t1); if (lane == 0) issue(ring_s + (stg ^ 1) * STAGE256_BYTES, nxt); }
    PFrag<NSET> P;
    if (nvalid == T) softmax_step<NSET, true>(A, sc, p.scale_log2, nvalid, lane, P);
    else softmax_step<NSET, false>(A, sc, p.scale_log2, nvalid, lane, P);
    if (cur.mv >= 0) v_tile<false, NSET>(A, vs, win, area, W, lane, P, nullptr, nvalid);
    else raw_accum<false, NSET>(A, p.raw + (long)raw_tile(cur.mv) * (T * D), nvalid, lane, P, nullptr);
    cur = nxt; stg ^= 1; it = t1;
    __syncwarp();                                      // every lane has read this stage before its next copies are issued
  }
  if (FLAT) {                                        // (not kept in registers across the main loop)
    // the merges write over the warp's barriers
    if (lane == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];\nmbarrier.inval.shared::cta.b64 [%1];\n" ::"r"(ring_s), "r"(ring_s + STAGE256_BYTES) : "memory");
    bh = __shfl_sync(FULLM, s_flat.pair, 0); split = __shfl_sync(FULLM, s_flat.split, 0); NS = __shfl_sync(FULLM, s_flat.ns, 0);
    b = bh / p.n_kv; kvh = bh % p.n_kv;
  } else NS = s_ns;
  // ---- merge the warps of the CTA, half by half: one partial per virtual head (2 * query head + half)
  if (__syncthreads_or(sum_warp(A))) sum_exact<true, true>(p, smem + T256_RING, bh, split, NS, FLAT ? s_flat.range : nullptr);
  else stage_warp(A, smem + T256_RING, G, warp, lane);
  __syncthreads();
  const int d = tid & 127;
  const long row0 = 2 * ((long)b * p.n_q + kvh * G);
  auto deliver = [&](long row, float L, float Ac) {
    const float v = L > 0.f ? Ac / L : 0.f;
    p.out[row * D + d] = __bfloat16_as_ushort(__float2bfloat16(v));
    if (p.out_f32) p.out_f32[row * D + d] = v;
  };
  float M[2 * NSET], Lc[2 * NSET], Ac[2 * NSET];      // of virtual heads tid / 128, 4 above, ..
#pragma unroll
  for (int i = 0; i < 2 * NSET; i++) {
    const int vg = (tid >> 7) + 4 * i;
    if (vg < 2 * G) merge_warps<ATT_WARPS / 2>(smem + T256_RING, 2, vg & 1, vg >> 1, d, M[i], Lc[i], Ac[i]);
  }
#pragma unroll
  for (int i = 0; i < 2 * NSET; i++) {
    const int vg = (tid >> 7) + 4 * i;
    if (vg >= 2 * G) continue;
    if (NS == 1) deliver(row0 + vg, Lc[i], Ac[i]);
    else {
      const long pidx = FLAT ? (long)(blockIdx.x + bh) * 2 * G + vg : (row0 + vg) * p.nsplit + split;
      if (d == 0) { p.pm[pidx] = M[i]; p.pl[pidx] = Lc[i]; }
      p.pa[pidx * D + d] = Ac[i];
    }
  }
  const bool last = NS > 1 && last_split(p.counters + bh, NS, &s_last);
  if (!FLAT && !last) return;
  if (FLAT) {
    for (int first = 0; last && first < 2 * G; first += 8) {
      __syncthreads();                                 // the area is used again
      merge_pieces<8>(p, smem + T256_RING, (long)(blockIdx.x - split + bh) * 2 * G + first, 1, 2 * G, min(8, 2 * G - first), NS, [&](int g, float, float L, float Ac) { deliver(row0 + first + g, L, Ac); });
    }
  } else {
#pragma unroll 1
    for (int vg = tid >> 7; vg < 2 * G; vg += ATT_THREADS / 128) {
      float Mv, Lv, Av;
      merge_splits<32>(p, (row0 + vg) * p.nsplit, 1, NS, d, Mv, Lv, Av);
      deliver(row0 + vg, Lv, Av);
    }
  }
  if (FLAT) {
    if (s_flat.share == 0) return;                   // (a plan of one piece per CTA: the walk would only find that out, 0.3 us later)
    __syncthreads();                                 // the shared memory is used again
  }
  } while (FLAT);
}

// Second half of the cross-GPU exchange as a launch of its own (the attention kernel was launched push-only): wait until
// every rank's rows of this exchange have arrived in this GPU's receive buffer, merge them, and advance the exchange number.
// One CTA per query head.  A row that has not arrived after X_WAIT_LIMIT polls sets *err and the head comes back as zeros.
__global__ void __launch_bounds__(128) exchange_merge_kernel(unsigned long long* const* x_recv, int* epoch, int* ticket, int* err, int rank, int world,
                                                              long rows_cap, uint16_t* __restrict__ out, float* __restrict__ out_f32) {
  const long qh = blockIdx.x; const int d = threadIdx.x;
  asm volatile("griddepcontrol.wait;" ::: "memory");                   // resident early, runs after the attention kernel has completed
  asm volatile("griddepcontrol.launch_dependents;" ::);
  const int ep = __ldcg(epoch);                                         // advanced only after every CTA has taken its ticket
  float v;
  const int bad = !x_merge_rows(x_recv[rank] + (long)(ep & 1) * world * rows_cap * 130, world, rows_cap, qh, d, (u32)ep + 1u, v);
  const int any_bad = __syncthreads_or(bad);
  if (any_bad) { v = 0.f; if (d == 0) atomicExch(err, 1); }
  if (out) out[qh * D + d] = __bfloat16_as_ushort(__float2bfloat16(v));
  if (out_f32) out_f32[qh * D + d] = v;
  __syncthreads();
  if (d == 0) {
    __threadfence();
    if (atomicAdd(ticket, 1) == (int)gridDim.x - 1) { *ticket = 0; __threadfence(); atomicAdd(epoch, 1); }
  }
}

// Merge partials: pm, pl [n_heads, n_parts], pa [n_heads, n_parts, 128] (m in natural-log units).
__global__ void __launch_bounds__(128) combine_kernel(const float* __restrict__ pm, const float* __restrict__ pl, const float* __restrict__ pa,
                                                       int n_parts, uint16_t* __restrict__ out, float* __restrict__ out_f32) {
  const long qh = blockIdx.x; const int d = threadIdx.x;
  float M = -CUDART_INF_F;
  for (int s = 0; s < n_parts; s++) M = fmaxf(M, pm[qh * n_parts + s]);
  float L = 0.f, Ac = 0.f;
  for (int s = 0; s < n_parts; s++) {
    const float ms = pm[qh * n_parts + s];
    const float f = (ms == -CUDART_INF_F) ? 0.f : __expf(ms - M);
    L += pl[qh * n_parts + s] * f; Ac += pa[(qh * n_parts + s) * D + d] * f;
  }
  const float v = L > 0.f ? Ac / L : 0.f;
  if (out) out[qh * D + d] = __bfloat16_as_ushort(__float2bfloat16(v));
  if (out_f32) out_f32[qh * D + d] = v;
}

// The same merge over packed partials: parts [n_parts][n_heads][130] = (m in natural-log units, l, acc[128]) per head, the
// layout an all-gather of the ranks' gaac_decode_attn_partial outputs produces.
__global__ void __launch_bounds__(128) combine_parts_kernel(const float* __restrict__ parts, long n_heads, int n_parts,
                                                             uint16_t* __restrict__ out, float* __restrict__ out_f32) {
  const long qh = blockIdx.x; const int d = threadIdx.x;
  float M = -CUDART_INF_F;
  for (int s = 0; s < n_parts; s++) M = fmaxf(M, parts[(s * n_heads + qh) * 130]);
  float L = 0.f, Ac = 0.f;
  for (int s = 0; s < n_parts; s++) {
    const float* pp = parts + (s * n_heads + qh) * 130;
    const float ms = pp[0];
    const float f = (ms == -CUDART_INF_F) ? 0.f : __expf(ms - M);
    L += pp[1] * f; Ac += pp[2 + d] * f;
  }
  const float v = L > 0.f ? Ac / L : 0.f;
  if (out) out[qh * D + d] = __bfloat16_as_ushort(__float2bfloat16(v));
  if (out_f32) out_f32[qh * D + d] = v;
}

// Rows of a batch from the longest to the shortest (ties by index): entry k = {row, its token count}, k < B.  Entry B says whether
// the order is worth using: {1, -} when the shortest non-empty row has less than 7/8 of the longest row's tokens, else {0, -}
// (rows of about equal length keep the grid's own numbering, which costs nothing).  One CTA; every thread finds the place of its
// own row by counting the rows that come before it.
constexpr int ORDER_MAX_ROWS = 1024;
__global__ void __launch_bounds__(ORDER_MAX_ROWS) row_order_kernel(const int* __restrict__ seq_lens, int B, int2* __restrict__ order) {
  __shared__ int len_s[ORDER_MAX_ROWS];
  __shared__ int mx_s, mn_s;
  const int t = threadIdx.x;
  asm volatile("griddepcontrol.wait;" ::: "memory");                   // resident early behind the previous kernel, as the attention kernels are
  asm volatile("griddepcontrol.launch_dependents;" ::);
  if (t == 0) { mx_s = 0; mn_s = 0x7fffffff; }
  if (t < B) len_s[t] = seq_lens[t];
  __syncthreads();
  if (t < B) {
    const int mine = len_s[t];
    atomicMax(&mx_s, mine);
    if (mine > 0) atomicMin(&mn_s, mine);
    int before = 0;
    for (int i = 0; i < B; i++) before += (len_s[i] > mine) || (len_s[i] == mine && i < t);
    order[before] = make_int2(t, mine);
  }
  __syncthreads();
  if (t == 0) order[B] = make_int2(mn_s < mx_s - (mx_s >> 3) ? 1 : 0, 0);
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
// Workspace = header | pm | pl | pa.  Header: the error word at byte 0, the split counters from byte 256.  The header has a
// fixed size for every B*n_q up to 16320, so the partials of a call never lie where the counters of a call of another shape
// do: a workspace zeroed once can be reused across batch sizes and split counts.
constexpr size_t WS_COUNTERS_OFF = 256, WS_MIN_HEADER = 64 << 10;
static size_t ws_header_bytes(int B, int n_q) { return std::max(WS_MIN_HEADER, WS_COUNTERS_OFF + align256(4 * (size_t)B * n_q)); }
static size_t ws_bytes_needed(int B, int n_q, int nsplit) {
  const size_t n = (size_t)B * n_q * nsplit;
  return ws_header_bytes(B, n_q) + align256(4 * n) * 2 + align256(4 * n * D) + align256(sizeof(int2) * ((size_t)B + 1));     // header | pm | pl | pa | row order
}
// Splits per row whose room the partials of a balanced launch fit into: n_kv * units * G = n_q * units rows.
static int share_splits(int B, int units) { return (units + B - 1) / B; }
static int carve_workspace(void* ws, size_t ws_bytes, int B, int n_q, int nsplit, AttnParams& p) {
  const size_t n = (size_t)B * n_q * nsplit;
  if (!ws || ws_bytes < ws_bytes_needed(B, n_q, nsplit)) return GAAC_E_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(ws) & 15) return GAAC_E_ALIGN;
  uint8_t* w = (uint8_t*)ws;
  p.err = (int*)w; p.counters = (int*)(w + WS_COUNTERS_OFF); w += ws_header_bytes(B, n_q);
  p.pm = (float*)w; w += align256(4 * n);
  p.pl = (float*)w; w += align256(4 * n);
  p.pa = (float*)w; w += align256(4 * n * D);
  p.order_buf = (int2*)w;
  return GAAC_OK;
}

static void launch_row_order(const int* seq_lens, int B, int2* order, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1); cfg.blockDim = dim3(ORDER_MAX_ROWS); cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = g_launch_overlap;
  cfg.attrs = at; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, row_order_kernel, seq_lens, B, order) != cudaSuccess) cudaGetLastError();     // the attention launch that follows reports
}

// Launch of an attention kernel, one CTA of ATT_THREADS per SM.  The permission for its shared memory is asked for once per kernel and device, not on every
// launch; where a launch fails with the permission believed to be there (it goes with a device reset), it is asked for again.
template <auto Kernel>
static int launch_big(const AttnParams& p, dim3 grid, int smem_bytes, cudaStream_t st, int team = 1) {
  static std::atomic<unsigned long long> allowed{0};                  // one bit per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return GAAC_E_LAUNCH; }
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(ATT_THREADS); cfg.dynamicSmemBytes = smem_bytes; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = g_launch_overlap;
  at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = (unsigned)team; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = team > 1 ? 2 : 1;
  bool asked = false;
  while (true) {
    if (asked || !(allowed.load(std::memory_order_relaxed) & bit)) {
      cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
      allowed.fetch_or(bit, std::memory_order_relaxed);
      asked = true;
    }
    if (cudaLaunchKernelEx(&cfg, Kernel, p) == cudaSuccess) return launch_status();
    cudaGetLastError();
    if (asked) return GAAC_E_LAUNCH;
    asked = true;
  }
}
template <bool PAGED, bool DUMP, int NSET, int MODE>
static int launch_attn_as(const AttnParams& p, cudaStream_t st) {
  const dim3 grid = MODE == FLAT_LINE ? dim3((unsigned)p.flat) : MODE == SHARED ? dim3((unsigned)p.n_kv, (unsigned)p.units) : dim3((unsigned)(p.B * p.n_kv), (unsigned)p.nsplit);
  return launch_big<decode_attn_kernel<PAGED, DUMP, NSET, MODE>>(p, grid, ATT_SMEM, st, MODE == TEAM ? p.nsplit : 1);
}
template <int NSET>
static int launch_attn256(const AttnParams& p, cudaStream_t st) {
  if (p.flat) return launch_big<paged256_attn_kernel<NSET, true>>(p, dim3((unsigned)p.flat), ATT256_SMEM, st);
  return launch_big<paged256_attn_kernel<NSET, false>>(p, dim3((unsigned)(p.B * p.n_kv), (unsigned)p.nsplit), ATT256_SMEM, st);
}
// Whether a launch may be made of teams: all of its clusters must fit the GPU at a time (15 of 8 or 7 CTAs, 22 of 6, 26 of 5, 33 of 4 on the one that this was measured on, since a cluster lies in one
// group of SMs; 16 rows in 8 ranges each take 11.7 us as clusters, 8.7 without), and they gain only where ranges are short.
template <bool PAGED, int NSET>
static int team_room(int nsplit) {
  static std::atomic<int> known[64][TEAM_MOST + 1];                   // clusters, and one
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 0; }
  int n = known[dev][nsplit].load(std::memory_order_relaxed) - 1;
  if (n < 0) {
    const auto kernel = decode_attn_kernel<PAGED, false, NSET, TEAM>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64, (unsigned)nsplit); cfg.blockDim = dim3(ATT_THREADS); cfg.dynamicSmemBytes = ATT_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = (unsigned)nsplit; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 0) {
      cudaGetLastError();
      return 0;                                      // (not known: asked again)
    }
    known[dev][nsplit].store(n + 1, std::memory_order_relaxed);
  }
  return n;
}
template <bool PAGED>
static bool team_ok(const AttnParams& p) {
  if (p.part || p.x_recv || p.row_order || p.nsplit < 2 || p.nsplit > TEAM_MOST) return false;
  if (!PAGED && !p.seq_len && ((p.S_uniform + T - 1) / T + p.nsplit - 1) / p.nsplit > TEAM_TILES) return false;
  // Clusters of 3 and of 5 need room for two more: launches of 44 or 45 and of 25 or 26 of them behind one another take up to 1.4 times as long as grids (45 rows of 21 tiles in 3 ranges 11.9 us
  // to 9.0; with another kernel between two of them 10.0 to 10.9), two fewer 0.9 times as long, as do the other sizes up to the last one.
  const int64_t spare = p.nsplit == 3 || p.nsplit == 5 ? 2 : 0;
  return (int64_t)p.B * p.n_kv + spare <= (p.G <= 4 ? team_room<PAGED, 1>(p.nsplit) : team_room<PAGED, 2>(p.nsplit));
}
template <bool PAGED, bool DUMP>
static int launch_attn(const AttnParams& p, cudaStream_t st) {
  if (!DUMP && p.flat) return p.G <= 4 ? launch_attn_as<PAGED, false, 1, FLAT_LINE>(p, st) : launch_attn_as<PAGED, false, 2, FLAT_LINE>(p, st);
  if (!DUMP && p.units) return p.G <= 4 ? launch_attn_as<PAGED, false, 1, SHARED>(p, st) : launch_attn_as<PAGED, false, 2, SHARED>(p, st);
  if (!DUMP && team_ok<PAGED>(p)) return p.G <= 4 ? launch_attn_as<PAGED, false, 1, TEAM>(p, st) : launch_attn_as<PAGED, false, 2, TEAM>(p, st);
  if (!DUMP && p.nsplit > 1 && (PAGED || p.seq_len)) return p.G <= 4 ? launch_attn_as<PAGED, false, 1, BOUND>(p, st) : launch_attn_as<PAGED, false, 2, BOUND>(p, st);
  return p.G <= 4 ? launch_attn_as<PAGED, DUMP, 1, GRID>(p, st) : launch_attn_as<PAGED, DUMP, 2, GRID>(p, st);
}

static int sm_count_of_current_device() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!cached[dev]) { int n = 0; if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) cached[dev] = n; else cudaGetLastError(); }
  return cached[dev];
}

static int share_wave(int B, int n_kv) { return std::max(B, sm_count_of_current_device() / n_kv); }

static bool exchange_ok(const gaac_exchange* x) {
  return x && x->recv && x->epoch && x->ticket && x->err && x->world >= 1 && x->world <= 64 && x->rank >= 0 && x->rank < x->world && x->rows_cap > 0;
}

// What the slot-layout entry points differ in.
struct SlotOut {
  void* out = nullptr; float* out_f32 = nullptr; float* part = nullptr;
  const gaac_exchange* x = nullptr; bool fused = false;
  int units = 0, flat = 0;
  void* dump_k = nullptr; void* dump_v = nullptr; int64_t dump_S = 0;
};
// Splits per row whose room the partials of a flat launch fit into, and whether the line's places can be counted in an int.
static int flat_splits(int B, int n_kv, int ctas) { return 1 + (int)(((int64_t)ctas + (int64_t)B * n_kv - 1) / ((int64_t)B * n_kv)); }
static bool flat_ok(int B, int n_kv, int ctas, int64_t longest) {
  return B > 0 && n_kv > 0 && ctas > 0 && ctas <= 1024 && longest >= 0 && longest < (1LL << 36) && (int64_t)B * n_kv < (1 << 24) && (int64_t)B * n_kv * (longest / T + 1 + FLAT_EXTRA) + ctas < 0x7FFFFFFFLL;
}

static int slot_attn(const gaac_side* K, const gaac_side* V, const void* q, const int32_t* slot, int B, int n_q, int n_kv, const int32_t* seq_len,
                     int64_t S_uniform, int64_t S_pad, float scale, int nsplit, const int32_t* tail_len, int tail_cap, int n_base_rows, void* ws, size_t ws_bytes,
                     const SlotOut& o, void* stream) {
  const gaac_exchange* x = o.x;
  if (!K || !V || !q || (!o.out && !o.part && !x) || (x && o.fused && !o.out)) return GAAC_E_ARG;
  if (x && !exchange_ok(x)) return GAAC_E_ARG;
  if (B <= 0 || n_q <= 0 || n_kv <= 0 || nsplit <= 0 || nsplit > 1024 || S_pad <= 0 || S_pad % T || n_base_rows <= 0) return GAAC_E_ARG;
  if (!seq_len && (S_uniform < 0 || S_uniform > S_pad)) return GAAC_E_ARG;
  if (n_q % n_kv || n_q / n_kv < 1 || n_q / n_kv > 8) return GAAC_E_UNSUPPORTED;
  if (x && (int64_t)B * n_q > x->rows_cap) return GAAC_E_ARG;
  // fused exchange: a CTA per (row, kv head) waits for the other GPUs inside the kernel, so every CTA of the grid must be
  // resident at once (one CTA per SM); larger grids use the push + gaac_exchange_merge pair
  if (x && o.fused && (int64_t)B * n_kv * nsplit > sm_count_of_current_device()) return GAAC_E_UNSUPPORTED;
  for (const gaac_side* s : {K, V}) {
    if (!s->sm || !s->codes || !s->flags || !s->tile_off || !s->ovf || !s->head_start || !s->base3 || !s->base4 || s->ovf_bytes < 0) return GAAC_E_ARG;
    if (!aligned16(s->sm) || !aligned16(s->codes) || !aligned16(s->flags) || (reinterpret_cast<uintptr_t>(s->ovf) & 3)) return GAAC_E_ALIGN;
    if (tail_len && (!s->tail || (reinterpret_cast<uintptr_t>(s->tail) & 3))) return GAAC_E_ARG;
  }
  if (tail_len && tail_cap <= 0) return GAAC_E_ARG;
  if (reinterpret_cast<uintptr_t>(q) & 3) return GAAC_E_ALIGN;
  if ((o.dump_k || o.dump_v) && (!o.dump_k || !o.dump_v || o.dump_S <= 0 || (reinterpret_cast<uintptr_t>(o.dump_k) & 3) || (reinterpret_cast<uintptr_t>(o.dump_v) & 3))) return GAAC_E_ARG;
  AttnParams p{};
  p.K = *K; p.V = *V; p.slot = slot; p.seq_len = seq_len; p.S_uniform = (int)S_uniform; p.tail_len = tail_len; p.tail_cap = tail_cap; p.S_pad = S_pad; p.n_base_rows = n_base_rows;
  p.q = (const uint16_t*)q; p.B = B; p.n_q = n_q; p.n_kv = n_kv; p.G = n_q / n_kv; p.scale_log2 = scale * LOG2E; p.nsplit = nsplit;
  p.out = (uint16_t*)o.out; p.out_f32 = o.out_f32; p.part = o.part; p.units = o.units; p.wave = o.units ? share_wave(B, n_kv) : 0; p.flat = o.flat;
  if (x) {
    p.x_recv = x->recv; p.x_epoch = x->epoch; p.x_ticket = x->ticket; p.x_err = x->err;
    p.x_rank = x->rank; p.x_world = x->world; p.x_rows_cap = x->rows_cap; p.x_fused = o.fused ? 1 : 0;
  }
  if (int e = carve_workspace(ws, ws_bytes, B, n_q, o.flat ? flat_splits(B, n_kv, o.flat) : o.units ? share_splits(B, o.units) : nsplit, p)) return e;
  if (o.dump_k) {
    p.dump_k = (uint16_t*)o.dump_k; p.dump_v = (uint16_t*)o.dump_v; p.dump_S = o.dump_S;
    return launch_attn<false, true>(p, (cudaStream_t)stream);
  }
  return launch_attn<false, false>(p, (cudaStream_t)stream);
}

static int paged_attn(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16, int B, int n_q, float scale,
                      int nsplit, int units, int flat, void* workspace, size_t workspace_bytes, void* out_bf16, float* out_f32, void* dump_k, void* dump_v, int64_t dump_S, void* stream) {
  if (!st || !bt || !seq_lens || !q_bf16 || !out_bf16 || !st->buf || !st->raw || !st->mt || !st->b3k || !st->b4k || !st->b3v || !st->b4v) return GAAC_E_ARG;
  if (B <= 0 || n_q <= 0 || st->n_kv <= 0 || nsplit <= 0 || nsplit > 1024 || bt_stride <= 0) return GAAC_E_ARG;
  if (n_q % st->n_kv || n_q / st->n_kv < 1 || n_q / st->n_kv > 8 || st->TS % 16 || st->TS != SLOT_OVF_OFF + st->ovf_slot) return GAAC_E_UNSUPPORTED;
  if (!aligned16(st->buf) || (reinterpret_cast<uintptr_t>(st->raw) & 3) || (reinterpret_cast<uintptr_t>(q_bf16) & 3)) return GAAC_E_ALIGN;
  if ((dump_k || dump_v) && (!dump_k || !dump_v || dump_S <= 0 || (reinterpret_cast<uintptr_t>(dump_k) & 3) || (reinterpret_cast<uintptr_t>(dump_v) & 3))) return GAAC_E_ARG;
  AttnParams p{};
  p.buf = st->buf; p.raw = (const uint16_t*)st->raw; p.mt = st->mt; p.bt = bt; p.bt_stride = bt_stride; p.TS = st->TS; p.ovf_slot = st->ovf_slot;
  p.b3k = st->b3k; p.b4k = st->b4k; p.b3v = st->b3v; p.b4v = st->b4v; p.seq_len = seq_lens;
  p.q = (const uint16_t*)q_bf16; p.B = B; p.n_q = n_q; p.n_kv = st->n_kv; p.G = n_q / st->n_kv; p.scale_log2 = scale * LOG2E; p.nsplit = nsplit;
  p.out = (uint16_t*)out_bf16; p.out_f32 = out_f32; p.part = nullptr; p.units = units; p.wave = units ? share_wave(B, st->n_kv) : 0; p.flat = flat;
  if (int e = carve_workspace(workspace, workspace_bytes, B, n_q, flat ? flat_splits(B, st->n_kv, flat) : units ? share_splits(B, units) : nsplit, p)) return e;
  if (dump_k) {
    p.dump_k = (uint16_t*)dump_k; p.dump_v = (uint16_t*)dump_v; p.dump_S = dump_S;
    return launch_attn<true, true>(p, (cudaStream_t)stream);
  }
  // ragged batches: CTAs are handed out longest row first (one small launch sorts the rows; its output is read by the attention
  // kernel after its dependency wait)
  if (!units && !flat && B > 1 && B <= ORDER_MAX_ROWS && (int64_t)B * st->n_kv * nsplit > sm_count_of_current_device()) {
    launch_row_order(seq_lens, B, p.order_buf, (cudaStream_t)stream);
    p.row_order = p.order_buf;
  }
  return launch_attn<true, false>(p, (cudaStream_t)stream);
}

}  // namespace gaac

using namespace gaac;

extern "C" void gaac_set_launch_overlap(int enabled) { g_launch_overlap = enabled ? 1 : 0; }

extern "C" size_t gaac_attn_workspace_bytes(int B, int n_q, int nsplit) {
  if (B <= 0 || n_q <= 0 || nsplit <= 0) return 0;
  return ws_bytes_needed(B, n_q, nsplit);
}

extern "C" size_t gaac_attn_workspace_header_bytes(int B, int n_q) {
  if (B <= 0 || n_q <= 0) return 0;
  return ws_header_bytes(B, n_q);
}

extern "C" int gaac_decode_attn(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                const int32_t* seq_len, int64_t S_pad, float scale, int nsplit, const int32_t* tail_len, int tail_cap,
                                int n_base_rows, void* workspace, size_t workspace_bytes, void* out_bf16, float* out_f32, void* stream) {
  if (!out_bf16 || !slot || !seq_len) return GAAC_E_ARG;
  SlotOut o; o.out = out_bf16; o.out_f32 = out_f32;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, 0, S_pad, scale, nsplit, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_decode_attn_balanced(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                         const int32_t* seq_len, int64_t S_pad, float scale, int units, const int32_t* tail_len, int tail_cap,
                                         int n_base_rows, void* workspace, size_t workspace_bytes, void* out_bf16, float* out_f32, void* stream) {
  if (!out_bf16 || !slot || !seq_len || B <= 0 || B > SHARE_MAX_ROWS || units < B || units - B + 1 > 1024) return GAAC_E_ARG;
  SlotOut o; o.out = out_bf16; o.out_f32 = out_f32; o.units = units;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, 0, S_pad, scale, units - B + 1, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_decode_attn_flat(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                     const int32_t* seq_len, int64_t S_pad, float scale, int ctas, const int32_t* tail_len, int tail_cap,
                                     int n_base_rows, void* workspace, size_t workspace_bytes, void* out_bf16, float* out_f32, void* stream) {
  if (!out_bf16 || !slot || !seq_len || !flat_ok(B, n_kv, ctas, S_pad)) return GAAC_E_ARG;
  SlotOut o; o.out = out_bf16; o.out_f32 = out_f32; o.flat = ctas;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, 0, S_pad, scale, 1, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_decode_attn_pages(const gaac_side* K, const gaac_side* V, const void* q_bf16, int B, int n_q, int n_kv, int64_t S, int64_t S_pad,
                                      float scale, int nsplit, int n_base_rows, void* workspace, size_t workspace_bytes, void* out_bf16, float* out_f32,
                                      float* part, const gaac_exchange* x, int fused, void* stream) {
  if ((out_bf16 != nullptr) + (part != nullptr) + (x != nullptr && !fused) != 1) return GAAC_E_ARG;      // exactly one destination
  SlotOut o; o.out = out_bf16; o.out_f32 = out_f32; o.part = part; o.x = x; o.fused = x && fused;
  return slot_attn(K, V, q_bf16, nullptr, B, n_q, n_kv, nullptr, S, S_pad, scale, nsplit, nullptr, 0, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_decode_attn_partial(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                        const int32_t* seq_len, int64_t S_pad, float scale, int nsplit, const int32_t* tail_len, int tail_cap,
                                        int n_base_rows, void* workspace, size_t workspace_bytes, float* part, void* stream) {
  if (!part || !slot || !seq_len) return GAAC_E_ARG;
  SlotOut o; o.part = part;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, 0, S_pad, scale, nsplit, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_combine(const float* pm, const float* pl, const float* pa, int64_t n_heads, int n_parts, void* out_bf16, float* out_f32, void* stream) {
  if (!pm || !pl || !pa || n_heads <= 0 || n_parts <= 0 || (!out_bf16 && !out_f32)) return GAAC_E_ARG;
  combine_kernel<<<(unsigned)n_heads, 128, 0, (cudaStream_t)stream>>>(pm, pl, pa, n_parts, (uint16_t*)out_bf16, out_f32);
  return launch_status();
}

extern "C" int gaac_decode_attn_push(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                     const int32_t* seq_len, int64_t S_pad, float scale, int nsplit, const int32_t* tail_len, int tail_cap,
                                     int n_base_rows, void* workspace, size_t workspace_bytes, const gaac_exchange* x, void* stream) {
  if (!x || !slot || !seq_len) return GAAC_E_ARG;
  SlotOut o; o.x = x;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, 0, S_pad, scale, nsplit, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_decode_attn_exchange(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                         const int32_t* seq_len, int64_t S_pad, float scale, int nsplit, const int32_t* tail_len, int tail_cap,
                                         int n_base_rows, void* workspace, size_t workspace_bytes, const gaac_exchange* x, void* out_bf16, float* out_f32,
                                         void* stream) {
  if (!x || !slot || !seq_len || !out_bf16) return GAAC_E_ARG;
  SlotOut o; o.x = x; o.fused = true; o.out = out_bf16; o.out_f32 = out_f32;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, 0, S_pad, scale, nsplit, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_exchange_merge(const gaac_exchange* x, int64_t n_heads, void* out_bf16, float* out_f32, void* stream) {
  if (!exchange_ok(x)) return GAAC_E_ARG;
  if (n_heads <= 0 || n_heads > x->rows_cap || (!out_bf16 && !out_f32)) return GAAC_E_ARG;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_heads); cfg.blockDim = dim3(128); cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = g_launch_overlap;
  cfg.attrs = at; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, exchange_merge_kernel, x->recv, x->epoch, x->ticket, x->err, x->rank, x->world,
                         (long)x->rows_cap, (uint16_t*)out_bf16, out_f32) != cudaSuccess) { cudaGetLastError(); return GAAC_E_LAUNCH; }
  return launch_status();
}

extern "C" int gaac_combine_parts(const float* parts, int64_t n_heads, int n_parts, void* out_bf16, float* out_f32, void* stream) {
  if (!parts || n_heads <= 0 || n_parts <= 0 || (!out_bf16 && !out_f32)) return GAAC_E_ARG;
  combine_parts_kernel<<<(unsigned)n_heads, 128, 0, (cudaStream_t)stream>>>(parts, (long)n_heads, n_parts, (uint16_t*)out_bf16, out_f32);
  return launch_status();
}

extern "C" int gaac_paged_decode_attn(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                                      int B, int n_q, float scale, int nsplit, void* workspace, size_t workspace_bytes,
                                      void* out_bf16, float* out_f32, void* stream) {
  return paged_attn(st, bt, bt_stride, seq_lens, q_bf16, B, n_q, scale, nsplit, 0, 0, workspace, workspace_bytes, out_bf16, out_f32, nullptr, nullptr, 0, stream);
}

extern "C" int gaac_paged_decode_attn_balanced(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                                               int B, int n_q, float scale, int units, void* workspace, size_t workspace_bytes,
                                               void* out_bf16, float* out_f32, void* stream) {
  if (B <= 0 || B > SHARE_MAX_ROWS || units < B || units - B + 1 > 1024) return GAAC_E_ARG;
  return paged_attn(st, bt, bt_stride, seq_lens, q_bf16, B, n_q, scale, units - B + 1, units, 0, workspace, workspace_bytes, out_bf16, out_f32, nullptr, nullptr, 0, stream);
}

extern "C" int gaac_paged_decode_attn_flat(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                                           int B, int n_q, float scale, int ctas, void* workspace, size_t workspace_bytes,
                                           void* out_bf16, float* out_f32, void* stream) {
  if (!st || bt_stride <= 0 || bt_stride > (1LL << 32) || !flat_ok(B, st->n_kv, ctas, bt_stride * T)) return GAAC_E_ARG;
  return paged_attn(st, bt, bt_stride, seq_lens, q_bf16, B, n_q, scale, 1, 0, ctas, workspace, workspace_bytes, out_bf16, out_f32, nullptr, nullptr, 0, stream);
}

static int paged_attn256(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                         int B, int n_q, float scale, int nsplit, int flat, void* workspace, size_t workspace_bytes,
                         void* out_bf16, float* out_f32, void* stream) {
  if (!st || !bt || !seq_lens || !q_bf16 || !out_bf16 || !st->buf || !st->raw || !st->mt || !st->b3k || !st->b4k || !st->b3v || !st->b4v) return GAAC_E_ARG;
  if (B <= 0 || n_q <= 0 || st->n_kv <= 0 || nsplit <= 0 || nsplit > 1024 || bt_stride <= 0) return GAAC_E_ARG;
  if (st->n_kv % 2) return GAAC_E_UNSUPPORTED;                                // half-heads come in pairs
  const int n_kv = st->n_kv / 2;                                              // 256-dim kv heads
  if (n_q % n_kv || n_q / n_kv < 1 || n_q / n_kv > 8 || st->TS % 16 || st->TS != SLOT_OVF_OFF + st->ovf_slot) return GAAC_E_UNSUPPORTED;
  if (!aligned16(st->buf) || (reinterpret_cast<uintptr_t>(st->raw) & 3) || (reinterpret_cast<uintptr_t>(q_bf16) & 3)) return GAAC_E_ALIGN;
  AttnParams p{};
  p.buf = st->buf; p.raw = (const uint16_t*)st->raw; p.mt = st->mt; p.bt = bt; p.bt_stride = bt_stride; p.TS = st->TS; p.ovf_slot = st->ovf_slot;
  p.b3k = st->b3k; p.b4k = st->b4k; p.b3v = st->b3v; p.b4v = st->b4v; p.seq_len = seq_lens;
  p.q = (const uint16_t*)q_bf16; p.B = B; p.n_q = n_q; p.n_kv = n_kv; p.G = n_q / n_kv; p.scale_log2 = scale * LOG2E; p.nsplit = nsplit;
  p.out = (uint16_t*)out_bf16; p.out_f32 = out_f32; p.flat = flat;
  if (int e = carve_workspace(workspace, workspace_bytes, B, 2 * n_q, flat ? flat_splits(B, n_kv, flat) : nsplit, p)) return e;     // one partial per (query head, half)
  return p.G <= 4 ? launch_attn256<1>(p, (cudaStream_t)stream) : launch_attn256<2>(p, (cudaStream_t)stream);
}

extern "C" int gaac_paged_decode_attn256(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                                         int B, int n_q, float scale, int nsplit, void* workspace, size_t workspace_bytes,
                                         void* out_bf16, float* out_f32, void* stream) {
  return paged_attn256(st, bt, bt_stride, seq_lens, q_bf16, B, n_q, scale, nsplit, 0, workspace, workspace_bytes, out_bf16, out_f32, stream);
}

extern "C" int gaac_paged_decode_attn256_flat(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                                              int B, int n_q, float scale, int ctas, void* workspace, size_t workspace_bytes,
                                              void* out_bf16, float* out_f32, void* stream) {
  if (!st || st->n_kv <= 0 || st->n_kv % 2 || bt_stride <= 0 || bt_stride > (1LL << 32) || !flat_ok(B, st->n_kv / 2, ctas, bt_stride * T)) return GAAC_E_ARG;
  return paged_attn256(st, bt, bt_stride, seq_lens, q_bf16, B, n_q, scale, 1, ctas, workspace, workspace_bytes, out_bf16, out_f32, stream);
}

// ---- test hooks: the same kernels, instantiated so that every rebuilt BF16 fragment is also written to memory
extern "C" int gaac_debug_decode_attn_rebuild(const gaac_side* K, const gaac_side* V, const void* q_bf16, const int32_t* slot, int B, int n_q, int n_kv,
                                              const int32_t* seq_len, int64_t S_uniform, int64_t S_pad, float scale, int nsplit, const int32_t* tail_len,
                                              int tail_cap, int n_base_rows, void* workspace, size_t workspace_bytes, void* out_bf16, float* out_f32,
                                              void* k_rebuilt, void* v_rebuilt, int64_t rebuilt_S, void* stream) {
  if (!out_bf16 || !k_rebuilt || !v_rebuilt) return GAAC_E_ARG;
  SlotOut o; o.out = out_bf16; o.out_f32 = out_f32; o.dump_k = k_rebuilt; o.dump_v = v_rebuilt; o.dump_S = rebuilt_S;
  return slot_attn(K, V, q_bf16, slot, B, n_q, n_kv, seq_len, S_uniform, S_pad, scale, nsplit, tail_len, tail_cap, n_base_rows, workspace, workspace_bytes, o, stream);
}

extern "C" int gaac_debug_team_room(int paged, int group, int nsplit) {
  if (nsplit < 2 || nsplit > TEAM_MOST || group < 1 || group > 8) return 0;
  return paged ? (group <= 4 ? team_room<true, 1>(nsplit) : team_room<true, 2>(nsplit)) : group <= 4 ? team_room<false, 1>(nsplit) : team_room<false, 2>(nsplit);
}

extern "C" int gaac_debug_paged_decode_attn_rebuild(const gaac_paged* st, const int32_t* bt, int64_t bt_stride, const int32_t* seq_lens, const void* q_bf16,
                                                    int B, int n_q, float scale, int nsplit, void* workspace, size_t workspace_bytes, void* out_bf16,
                                                    float* out_f32, void* k_rebuilt, void* v_rebuilt, int64_t rebuilt_S, void* stream) {
  if (!k_rebuilt || !v_rebuilt) return GAAC_E_ARG;
  return paged_attn(st, bt, bt_stride, seq_lens, q_bf16, B, n_q, scale, nsplit, 0, 0, workspace, workspace_bytes, out_bf16, out_f32, k_rebuilt, v_rebuilt, rebuilt_S, stream);
}
