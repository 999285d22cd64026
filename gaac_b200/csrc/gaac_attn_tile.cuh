// Warp-level pieces of the fused decode attention: asynchronous copies, the rebuild of a compressed 16-token tile into tensor-core
// fragments, the score and value products and the online softmax step.  Used by the kernels of gaac_attn.cu.
//
// What bounds them, measured on a B200 at batch 1, 32 query / 8 kv heads, 65536 tokens, 47.1 us: 950 warp instructions per (K tile + V tile) at 0.65 per cycle and scheduler, with
// four warps to a scheduler; 430 of them on the ALU (59 % of its cycles), 279 wavefronts of shared memory, DRAM 44 %.  A warp issues every 6.1 cycles and spends, of these, 1.1 waiting for a
// result of fixed latency, 1.1 ready but not chosen, 1.0 on shared memory, 0.7 on a busy pipe (the ALU), 0.3 at barriers, 0.3 on global memory: instructions first, then latency, since a
// third of the issue slots finds no warp ready.  More warps do not help (gaac_attn.cu: 18 or 20 at 96 registers).  Timing-only builds of a form of 51 us: without the raw groups 47,
// without any of plan_tile 39, with the payload read without bank conflicts 51, with no work on the tiles at all 34.  What did not help: moving shifts from the ALU to the FMA pipe, fewer
// or longer chains at the same count of instructions, warps of their own for plan_tile or for the copies.
//
// Head columns.  The tensor-core tile has 8 columns.  Query heads are handled in sets of four (NSET = 1 for a GQA group of up to
// 4, 2 for 5..8); lane j of a quad works for head 4 * set + j throughout:
//   scores  S^T[16 tok x 8] = K[16 x 128] . Q^T : column 2j = head j of set 0, column 2j + 1 = head j of set 1 (zero without it)
//   values, one set: a rebuilt word holds TWO channels of one token, so O^T += V^T . P^T contracts over (token, channel parity) and column
//           2j + parity takes (P, 0) or (0, P): the words go into the product as they were decoded, with no transpose, and each lane
//           gets both channels of its own head.  16 products per tile, as many as a transposed form has for 8 heads
//   values, two sets: the columns are the heads, as for the scores, and the words of two tokens are transposed by 32 byte permutes per tile.  The form
//           above takes 32 products and 16 registers of weights where this takes 16 and 4, and was slower: group of 8, 8 kv heads, 65536
//           tokens 67.1 us, 64.4 with it; paged 32768 40.1 -> 38.7; head_dim 256, 8 x 8000: 119 -> 111.  Words of two tokens made by the rebuild itself, with its last
//           permutes taking both: 64 x 32768 189.6 -> 189.4 and 32 bytes of spills, so not kept
#pragma once
#include <cuda_bf16.h>
#include <math_constants.h>
#include "gaac_lane.cuh"

namespace gaac {

constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

__device__ __forceinline__ void mma16816(float& c0, float& c1, float& c2, float& c3, u32 a0, u32 a1, u32 a2, u32 a3, u32 b0, u32 b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c0), "+f"(c1), "+f"(c2), "+f"(c3) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16816(float* c, u32 a0, u32 a1, u32 a2, u32 a3, u32 b0, u32 b1) { mma16816(c[0], c[1], c[2], c[3], a0, a1, a2, a3, b0, b1); }
// ---- bulk asynchronous copies (TMA engine, no tensor map): global -> shared, completion counted in bytes on an mbarrier.
// Both addresses are 16-byte aligned and the size is a multiple of 16 at every call site.
__device__ __forceinline__ void mbar_init(u32 mbar, u32 count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mbar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(u32 mbar, u32 bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(u32 dst, const void* src, u32 bytes, u32 mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}
// The same issued by one lane of a converged warp.  Executed by the whole warp with operands that are uniform, so that they go straight into the copy instruction's
// uniform registers: behind a branch on the lane number the compiler picks them up lane by lane in a loop.
__device__ __forceinline__ void warp_expect_tx(u32 mbar, u32 bytes) {
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n @p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void warp_add_tx(u32 mbar, u32 bytes) {
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n @p mbarrier.expect_tx.shared::cta.b64 [%0], %1;\n}\n" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void warp_g2s(u32 dst, const void* src, u32 bytes, u32 mbar) {
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n @p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n}\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}
// Bounded wait for a phase of the barrier: false when it gave up (the copies of a stage normally land within microseconds;
// the bound is there so that a lost copy can never hang the GPU).
constexpr int MBAR_WAIT_LIMIT = 1 << 22;
__device__ __forceinline__ bool mbar_wait(u32 mbar, u32 parity) {
  for (int it = 0; it < MBAR_WAIT_LIMIT; it++) {
    u32 ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
    if (ok) return true;
  }
  return false;
}
// The same for the phase that belongs to use number `use` of the barrier, as a word in shared memory says: it is `use` << 4 | flags when the phase has begun.
__device__ __forceinline__ bool mbar_wait_use(u32 mbar, u32 parity, u32 word, u32 use, u32& flags) {
  for (int it = 0; it < MBAR_WAIT_LIMIT; it++) {
    u32 v, ok;
    asm volatile("ld.relaxed.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(word) : "memory");
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
    flags = v & 15u;
    if (ok && v >> 4 == use) return true;
  }
  return false;
}
// A counter in shared memory, incremented by lane 0; its former value there.  The address counts the lane in: where it is the same in all lanes the compiler adds up a warp's
// increments first (votes, population counts, the lane masks out of special registers), some 10 instructions and their latency twice per tile for the one lane that there is.  65536 tokens
// 49.0 -> 47.7 us, 64 x 32768 195.7 -> 190.7, paged 16 x 4096..65536 391 -> 383 (steps in graphs); without a branch, but with one address, nothing.
template <bool ORDERED> __device__ __forceinline__ int lane_inc(u32 at, int lane) {
  int old = 0;
  if (ORDERED) asm volatile("{\n .reg .pred p;\n setp.eq.s32 p, %2, 0;\n @p atom.acq_rel.cta.shared::cta.inc.u32 %0, [%1], 0xffffffff;\n}\n" : "+r"(old) : "r"(at + 4u * (u32)lane), "r"(lane) : "memory");
  else asm volatile("{\n .reg .pred p;\n setp.eq.s32 p, %2, 0;\n @p atom.relaxed.cta.shared::cta.inc.u32 %0, [%1], 0xffffffff;\n}\n" : "+r"(old) : "r"(at + 4u * (u32)lane), "r"(lane) : "memory");
  return old;
}
__device__ __forceinline__ float fast_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// What a warp needs to know of a tile besides its staged bytes.  Slot layout: offsets of the tile's escape bytes inside the head's
// escape bytes.  Paged layout: the mode-table entries (>= 0: compressed slot, < 0: bit-complement of a raw tile of the pool).
struct TileMeta { int mk, mv; };

// ---- running state of one warp.  acc[set][mt][c] = O[head 4 * set + j][channel 8 * acc_channel(mt, c) + r]; m, l in the exp2 domain, l summed over
// this lane's tokens only.  Words mt and c >> 1 hold elements that are four apart.
__host__ __device__ constexpr int acc_channel(int mt, int c) { return 8 * (mt >> 1) + 2 * (mt & 1) + (c >> 1) + 4 * (c & 1); }
template <int NSET> struct WarpAcc {
  float acc[NSET][4][4];
  float m[NSET], l[NSET];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int s = 0; s < NSET; s++) {
      m[s] = -CUDART_INF_F; l[s] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; i++) acc[s][i][0] = acc[s][i][1] = acc[s][i][2] = acc[s][i][3] = 0.f;
    }
  }
};

// Q^T B-fragments of the score product.  Lane (j, r) provides column r = head 4 * (r & 1) + (r >> 1), zero where the group has no such head; the words pair the
// channels that a rebuilt word pairs: product 2g has c and c + 16, then c + 1 and c + 17 (c = 32g + 2j), product 2g + 1 the same 8 channels on.
struct QFrag { u32 qa[8][2]; };
__device__ __forceinline__ int q_head(int r) { return 4 * (r & 1) + (r >> 1); }
__device__ __forceinline__ void load_q(QFrag& Q, const uint16_t* q0, long head_stride, int G, int lane) {
  const int j = lane & 3, h = q_head(lane >> 2);
  const uint16_t* qp = q0 + (h < G ? h : 0) * head_stride;
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const uint16_t* c = qp + 32 * (s >> 1) + 2 * j + 8 * (s & 1);
    const u32 a = h < G ? *reinterpret_cast<const u32*>(c) : 0u, b = h < G ? *reinterpret_cast<const u32*>(c + 16) : 0u;
    Q.qa[s][0] = prmt(a, b, 0x5410); Q.qa[s][1] = prmt(a, b, 0x7632);
  }
}

// Weights of one tile as B-fragments of the value product.  A weight enters as the sum of two BF16 numbers, its rounded value (hi) and the rounded
// remainder (lo), which brings its relative error to 2^-16.  One set: [0]: places 0 (b0) and 1 (b1) of slot_token, [1]: places 2 and 3.  Two: [0]:
// places 0, 1, [1]: places 2, 3.
template <int NSET> struct PFrag;
template <> struct PFrag<1> { u32 hi[2][2], lo[2][2]; };
template <> struct PFrag<2> { u32 hi[2], lo[2]; };
__device__ __forceinline__ u32 pack_bf16(float lo, float hi) { __nv_bfloat162 x = __floats2bfloat162_rn(lo, hi); return *reinterpret_cast<u32*>(&x); }
// what the rounding of a pair dropped, which fp32 holds exactly, rounded in turn
__device__ __forceinline__ u32 pack_rest(float lo, float hi, u32 rounded) { return pack_bf16(lo - __uint_as_float(rounded << 16), hi - __uint_as_float(rounded & 0xFFFF0000u)); }

// Token of the lane's place i in the value product: places 0, 1 are tokens 2j, 2j + 1 and places 2, 3 the same 8 on, for lanes j = 2, 3 the other way round.  A lane's four
// tokens lie 64 bytes from the next lane's in a staged V tile; read in one order by all lanes they meet in a quarter of the banks, so that half of them start at
// the other end.  (0.6 % of the kernel.)
__device__ __forceinline__ int slot_token(int j, int i) { return 2 * j + (i & 1) + 8 * ((i >> 1) ^ (j >> 1)); }
// p0, p8: this lane's weights of tokens r and r + 8 for head j of each set.
// One set: as column r of the value product the lane needs those of head r >> 1 for the tokens of its places, in the low (parity 0) or high
// (parity 1) half of a word whose other half is zero.
__device__ __forceinline__ void put_weights(PFrag<1>& P, const float (&p0)[1], const float (&p8)[1], int lane) {
  const int j = lane & 3, r = lane >> 2, src = 8 * j + (r >> 1);
  const bool sw = j >= 2;
  const u32 selA = (r & 1) ? 0x1044u : 0x4410u, selB = (r & 1) ? 0x3244u : 0x4432u, sel0 = sw ? selB : selA, sel8 = sw ? selA : selB;
  const u32 H = pack_bf16(p0[0], p8[0]), L = pack_rest(p0[0], p8[0], H);
  const u32 ha = __shfl_sync(FULLM, H, src), hb = __shfl_sync(FULLM, H, src + 4), la = __shfl_sync(FULLM, L, src), lb = __shfl_sync(FULLM, L, src + 4);
  P.hi[0][0] = prmt(ha, 0u, sel0); P.hi[0][1] = prmt(hb, 0u, sel0); P.hi[1][0] = prmt(ha, 0u, sel8); P.hi[1][1] = prmt(hb, 0u, sel8);
  P.lo[0][0] = prmt(la, 0u, sel0); P.lo[0][1] = prmt(lb, 0u, sel0); P.lo[1][0] = prmt(la, 0u, sel8); P.lo[1][1] = prmt(lb, 0u, sel8);
}
// Two: column r is head r >> 1 of set r & 1, its words hold two tokens.
__device__ __forceinline__ void put_weights(PFrag<2>& P, const float (&p0)[2], const float (&p8)[2], int lane) {
  const int j = lane & 3, r = lane >> 2, src = 8 * j + (r >> 1);
  const u32 sel = (r & 1) ? 0x7632u : 0x5410u;
  const bool sw = lane >= 16;                          // the lanes that read from this one have their places the other way round
  const float x0 = sw ? p8[0] : p0[0], x1 = sw ? p8[1] : p0[1], y0 = sw ? p0[0] : p8[0], y1 = sw ? p0[1] : p8[1];
  const u32 h0 = pack_bf16(x0, x1), h8 = pack_bf16(y0, y1), l0 = pack_rest(x0, x1, h0), l8 = pack_rest(y0, y1, h8);
  const u32 a0 = __shfl_sync(FULLM, h0, src), b0 = __shfl_sync(FULLM, h0, src + 4), a8 = __shfl_sync(FULLM, h8, src), b8 = __shfl_sync(FULLM, h8, src + 4);
  const u32 c0 = __shfl_sync(FULLM, l0, src), d0 = __shfl_sync(FULLM, l0, src + 4), c8 = __shfl_sync(FULLM, l8, src), d8 = __shfl_sync(FULLM, l8, src + 4);
  P.hi[0] = prmt(a0, b0, sel); P.hi[1] = prmt(a8, b8, sel); P.lo[0] = prmt(c0, d0, sel); P.lo[1] = prmt(c8, d8, sel);
}

// Online softmax on the score fragment.  The running maximum is only raised (and the accumulators rescaled) when some score of the
// tile exceeds it by more than RESCALE_TAU in the exp2 domain; otherwise the tile is weighted against the stale maximum, so P stays
// below 2^RESCALE_TAU.  Sums and accumulators are fp32 and P keeps its relative rounding, so the result is as exact as with the true
// maximum, and the common tile needs no cross-lane reduction, no rescale factor and no accumulator multiply.
constexpr float RESCALE_TAU = 16.f;
template <int NSET, bool FULL_TILE>
__device__ __forceinline__ void softmax_step(WarpAcc<NSET>& A, const float* sc, float scale_log2, int nvalid, int lane, PFrag<NSET>& P) {
  const int r = lane >> 2;
  float s0[NSET], s8[NSET];
  bool over = false;
#pragma unroll
  for (int s = 0; s < NSET; s++) {
    s0[s] = FULL_TILE || r < nvalid ? sc[s] * scale_log2 : -CUDART_INF_F;             // a full tile needs no token masks
    s8[s] = FULL_TILE || r + 8 < nvalid ? sc[2 + s] * scale_log2 : -CUDART_INF_F;
    over |= fmaxf(s0[s], s8[s]) > A.m[s] + RESCALE_TAU;
  }
  if (__any_sync(FULLM, over)) {
#pragma unroll
    for (int s = 0; s < NSET; s++) {
      float mt = fmaxf(s0[s], s8[s]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) mt = fmaxf(mt, __shfl_xor_sync(FULLM, mt, o));
      const float mn = fmaxf(A.m[s], mt), al = (mn == -CUDART_INF_F) ? 0.f : fast_exp2(A.m[s] - mn);
      A.l[s] *= al; A.m[s] = mn;
#pragma unroll
      for (int i = 0; i < 4; i++) { A.acc[s][i][0] *= al; A.acc[s][i][1] *= al; A.acc[s][i][2] *= al; A.acc[s][i][3] *= al; }
    }
  }
  float p0[NSET], p8[NSET];
#pragma unroll
  for (int s = 0; s < NSET; s++) {
    const float mu = fmaxf(A.m[s], -1e30f);                                          // a maximum of -inf (nothing seen yet) must not produce inf - inf
    p0[s] = fast_exp2(s0[s] - mu); p8[s] = fast_exp2(s8[s] - mu);
    A.l[s] += p0[s] + p8[s];
  }
  put_weights(P, p0, p8, lane);
}

// Value product of two words (2 * mt and the next) of the lane's four tokens (2j, 2j + 1, 2j + 8, 2j + 9).
__device__ __forceinline__ void pv_words(WarpAcc<1>& A, int mt, const u32 (&w0)[4], const u32 (&w1)[4], const PFrag<1>& P) {
  mma16816(A.acc[0][mt], w0[0], w1[0], w0[1], w1[1], P.hi[0][0], P.hi[0][1]);
  mma16816(A.acc[0][mt], w0[0], w1[0], w0[1], w1[1], P.lo[0][0], P.lo[0][1]);
  mma16816(A.acc[0][mt], w0[2], w1[2], w0[3], w1[3], P.hi[1][0], P.hi[1][1]);
  mma16816(A.acc[0][mt], w0[2], w1[2], w0[3], w1[3], P.lo[1][0], P.lo[1][1]);
}
__device__ __forceinline__ void pv_words(WarpAcc<2>& A, int mt, const u32 (&w0)[4], const u32 (&w1)[4], const PFrag<2>& P) {
#pragma unroll
  for (int h = 0; h < 2; h++) {                      // the two channels of word i + h are rows r and r + 8
    const u32 (&w)[4] = h ? w1 : w0;
    const u32 a0 = prmt(w[0], w[1], 0x5410), a1 = prmt(w[0], w[1], 0x7632), a2 = prmt(w[2], w[3], 0x5410), a3 = prmt(w[2], w[3], 0x7632);
    float &c0 = A.acc[0][mt][2 * h], &c1 = A.acc[1][mt][2 * h], &c2 = A.acc[0][mt][2 * h + 1], &c3 = A.acc[1][mt][2 * h + 1];
    mma16816(c0, c1, c2, c3, a0, a1, a2, a3, P.hi[0], P.hi[1]);
    mma16816(c0, c1, c2, c3, a0, a1, a2, a3, P.lo[0], P.lo[1]);
  }
}

// ---- CTA tables and the stage layout
// Escape bytes staged per tile and kind (the slot layout's tiles of a stage share theirs); longer tiles read theirs from global memory, at half
// the speed.  256 is every group of a tile promoted, a base table that is off by a few exponents.  With 192: 32768 tokens, 8 kv heads, all groups
// promoted 48.5 us, now 36.1 (33.6 with tables that fit); paged, half of the channels off: 42.1, now 38.3.
constexpr int ESC_WIN = 256;
constexpr int PSLOT = SLOT_OVF_OFF + ESC_WIN + 16;          // staged bytes of a paged tile slot, at most
// What a planned tile pair has in shared memory (its segment area): segment words of K and of V, [row][quarter of a row], 8 bytes per segment, then the entries of
// its raw groups.  PATCH_MAX: raw groups of a tile pair (of 512) that have room (what shared memory leaves); a pair with more takes the plain decoder.
constexpr int PATCH_MAX = 62, SEG_K = 0, SEG_V = 64 * 8, SEG_PATCH = 2 * SEG_V;
constexpr int AREA_BYTES = SEG_PATCH + 8 * PATCH_MAX;
// Addend table: entry NO_ESC (zero) and entries 256 + byte, 8 bytes each; segment table: 256 entries of 8 bytes
constexpr int ADDEND_BYTES = 8 + 257 * 8, SEGTAB_BYTES = 256 * 8;

// Shared-memory addresses that do not change from tile to tile: entry 0 of the addend table (which begins with entry NO_ESC), the segment table, the base words
// (K, then V).  Segment areas lie behind the tables.
struct AttnView { u32 addends, segs, bases; };
// Fill the tables with threads t = 0 .. 255.  at: ADDEND_BYTES + SEGTAB_BYTES on a 16-byte boundary; returned: the addresses of the view.
__device__ __forceinline__ void fill_attn_tables(uint8_t* at, int t) {
  const u32x2 x = pair_addends((u32)t), s = segment_entry((u32)t);
  reinterpret_cast<uint2*>(at + 16)[t] = make_uint2(x.x, x.y);
  reinterpret_cast<uint2*>(at + ADDEND_BYTES)[t] = make_uint2(s.x, s.y);
  if (t == 0) reinterpret_cast<uint2*>(at + 8)[0] = make_uint2(0u, 0u);
}
__device__ __forceinline__ AttnView attn_view(u32 tables, u32 bases) { return AttnView{tables + 16 - 256 * 8, tables + ADDEND_BYTES, bases}; }
// Base words of a side: group t of 16 by thread t, 16 bytes each.  K: lane class j, group g at 80 * j + 16 * g, where the four groups that a load reads at a time lie in different
// banks (at 64 * j two by two in the same: 298 cycles of the shared-memory pipe per tile pair, now 282;  65536 tokens 52.5 us, now 51.9);  V: class r, group g at 32 * r + 16 * g behind them.
constexpr int PAIR_BASES_V = 16 * (16 + 3), PAIR_BASES_BYTES = PAIR_BASES_V + 16 * 16;
template <bool VSIDE>
__device__ __forceinline__ void fill_pair_bases(uint8_t* bases, const uint8_t* b3, const uint8_t* b4, int t) {
  const u32x4 w = pair_base_words<VSIDE>(b3, b4, t);
  *reinterpret_cast<uint4*>(bases + (VSIDE ? PAIR_BASES_V : 0) + 16 * (VSIDE ? t : t + (t >> 2))) = make_uint4(w.x, w.y, w.z, w.w);
}

// One side (K or V) of a staged tile; glob = its escape bytes in global memory.
struct SideView { const uint8_t *sm, *cd, *glob; };
// ---- escape bytes of a tile pair.  A segment is four neighbouring groups of a row, one byte of its tag word.  It is expanded into a word per two groups with a
// 16-bit index into the addend table for each (gaac_tile.h), which go to the tile pair's segment area, where the lanes that rebuild the groups find them.  A side whose escape bytes are not all staged has {tag byte | position << 16} there instead, and
// its escape bytes are read from global memory.
// Once per segment, because a group's share of it (tag bits, position, byte, table address) cost 10 of the 37 instructions of its rebuild.

// prmt with a selector that is not known: the intrinsic masks it first.
__device__ __forceinline__ u32 permute(u32 a, u32 b, u32 sel) { u32 d; asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel)); return d; }
// One step of an inclusive scan over each half of a warp (scan_step over all of it).
__device__ __forceinline__ void scan_step16(u32& v, int d) {
  asm volatile("{\n .reg .pred p;\n .reg .u32 t;\n shfl.sync.up.b32 t|p, %0, %1, 0x1000, 0xffffffff;\n @p add.u32 %0, %0, t;\n}\n" : "+r"(v) : "r"(d));
}
// Make the segment area of a tile pair.  Lane l has row l & 15 of K (l < 16) or of V.  live: the lane's side is compressed; fl, esc: shared-memory addresses of its
// tag words and of its escape bytes, of which `avail` are staged.  Returned: bit 0 / 1: those of K / V are all staged (and the staged sides have no more than `room` raw
// groups, which have their entries, 8 bytes each, behind the segment words; the other groups of raw_items need none).
// Bound by its instructions, 282 of 1052 per tile pair before, about 200 of 950 now, and by its chain of latencies; hence a scan over 16 rows and not over 64 segments, and sizes from the tag words
// while the segment table answers.  The scan counts the raw groups along with the escape bytes, so that a row knows its entries' places and takes its items without asking the
// others.  The raw groups, 4 of 512, took half of it (147 instructions: 1.8 trips of a loop in which both kinds of item lay on either side of a branch; a timing-only build without that loop 51.3 -> 46.6 us).
// Now each kind has a loop of its own, from the last item to the first, where the mask of what lies below an item also takes it off, and one vote asks whether everything is staged and
// has room, which it nearly always has.  65536 tokens 51.4 -> 49.8 us, 64 x 32768 205.3 -> 199.3, paged 16 x 4096..65536 422 -> 406 (steps in graphs).
__device__ __forceinline__ int plan_tile(bool live, u32 fl_at, u32 esc, int avail, const AttnView& w, u32 area, u32 room, int lane) {
  const u32 fl = live ? lds_u32(fl_at + 4u * (lane & 15)) : 0u;
  const u32 ones = (u32)popc(fl & 0x55555555u), own_raws = (u32)popc(fl & 0xAAAAAAAAu), own = mad_k<65540u>(own_raws, ones);            // escape bytes | raw groups << 16
  const u32x2 e[4] = {lds_u64(mad_byte<0, 8u>(fl, w.segs)), lds_u64(mad_byte<1, 8u>(fl, w.segs)), lds_u64(mad_byte<2, 8u>(fl, w.segs)), lds_u64(mad_byte<3, 8u>(fl, w.segs))};
  u32 sum = own;
  scan_step16(sum, 1); scan_step16(sum, 2); scan_step16(sum, 4); scan_step16(sum, 8);
  const u32 end = sum & 0xFFFFu, k_raws = __shfl_sync(FULLM, sum, 15) >> 16, mine = area + 32u * lane;
  u32 past = (sum >> 16) + (lane >= 16 ? k_raws : 0u), pos = (sum - own) & 0xFFFFu;           // places behind the row's entries, those of K first;  the row's first escape byte
  int staged = 3;
  bool fast = true;
  if (__any_sync(FULLM, (live && (int)end > avail) || past > room)) {
    const u32 over = __ballot_sync(FULLM, live && (int)end > avail);
    staged = ((over & 0xFFFFu) ? 0 : 1) | ((over >> 16) ? 0 : 2);
    if (lane >= 16 && !(staged & 1)) past -= k_raws;         // (K's side needs no entries)
    fast = (staged >> (lane >> 4)) & 1;
    if (__any_sync(FULLM, fast && past > room)) { staged = 0; fast = false; }
    if (!fast) {                                     // {tag byte | position << 16}
#pragma unroll
      for (int q = 0; q < 4; q++) { sts_u64(mine + 8u * q, ((fl >> (8 * q)) & 0xFFu) | pos << 16, 0u); pos += e[q].x >> 16; }
    }
  }
  if (fast) {
    const u32 at = live ? esc + pos : area;
    u32 a = at, four[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const u32 lo = lds_u32(a & ~3u), hi = lds_u32((a & ~3u) + 4u);
      four[q] = __funnelshift_r(lo, hi, 8u * a);                             // (the shift counts modulo 32)
      a += e[q].x >> 16;
    }
#pragma unroll
    for (int q = 0; q < 4; q += 2)
      sts_u128(mine + 8u * q, permute(four[q], SEG_CONST, e[q].x), permute(four[q], SEG_CONST, e[q].y), permute(four[q + 1], SEG_CONST, e[q + 1].x), permute(four[q + 1], SEG_CONST, e[q + 1].y));
    // the raw groups, and the promoted ones behind a raw one of their segment, from the last to the first:  bit: lower tag bit of the group, 2 * group
    u32 raws = (fl >> 1) & fl & 0x55555555u;
    u32 behind = raw_items(fl) & ~raws;
    u32 index = ((area + SEG_PATCH - w.addends) >> 3) + past;
    const u32 side = w.bases + (lane >= 16 ? PAIR_BASES_V : 0), skew = lane >= 16 ? 0u : 16u;
    while (raws) {
      u32 bit; asm("bfind.u32 %0, %1;" : "=r"(bit) : "r"(raws));
      const u32 below = ~(0xFFFFFFFFu << bit);
      raws &= below; index--;
      const u32 pl = at + esc_below(fl, below);
      const u32x4 bw = lds_u128(side + 8u * bit + skew * (bit >> 3));
      const u32x2 x = pair_payload(__funnelshift_r(lds_u32(pl & ~3u), lds_u32((pl & ~3u) + 4u), 8u * pl), lds_u8(pl + 4u));
      const u32 m = index >> 8;
      sts_u64(w.addends + 8u * index, x.x - bw.x - m * bw.z, x.y - bw.y - m * bw.w);          // the upper bits of the exponents, less what the decoder will add to them
      sts_u16(mine + bit, index);
    }
    while (behind) {
      u32 bit; asm("bfind.u32 %0, %1;" : "=r"(bit) : "r"(behind));
      const u32 below = ~(0xFFFFFFFFu << bit);
      behind &= below;
      sts_u16(mine + bit, 256u + lds_u8(at + esc_below(fl, below)));
    }
  }
  __syncwarp();
  return staged;
}

// One group whose escape bytes are staged: H = half of the segment word with its index.  The addend's address and the group's m (byte 1 of the index) come out of the word by a dot product
// each: by shifts and masks they took 16 instructions more per tile pair, all of them on the ALU, which is the busiest pipe.  In graphs: 65536 tokens 53.4 -> 52.6 us, steps of 64 x 32768
// 211 -> 207 and of 16 x 4096..65536 paged 424 -> 421 (their public calls 440 -> 437, which is within the spread of runs).  (Not so the shifts and additions of rebuild_pairs as multiply-adds: 52.6 -> 52.6 and 53.7.)
template <int H> __device__ __forceinline__ void decode_staged(u32 sm_lo, u32 sm_hi, u32 u, u32 word, const AttnView& w, const u32x4& bw, u32 out[4]) {
  rebuild_pairs(sm_lo, sm_hi, u, mad_byte<2 * H + 1, 1u>(word, 0u), bw, lds_u64(mad_half<H, 8u>(word, w.addends)), out);
}
// One group whose escape bytes are read from global memory at glob[pos]; tg = its tag in the low bits.  pos advances past them.
__device__ __forceinline__ void decode_plain(u32 sm_lo, u32 sm_hi, u32 u, u32 tg, u32& pos, const uint8_t* glob, const AttnView& w, const u32x4& bw, u32 out[4]) {
  const u32 m = tg & 1u;
  u32x2 x = lds_u64(w.addends + 8u * (m ? 256u + glob[pos] : NO_ESC));
  if (tg & 2u) {
    const uint8_t* p = glob + pos;
    const u32* a = reinterpret_cast<const u32*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3);
    x = pair_raw_addends(a[0], a[1], 8u * (u32)(reinterpret_cast<uintptr_t>(p) & 3));
    x.x -= bw.x + bw.z; x.y -= bw.y + bw.w;
    pos += 4;
  }
  pos += m;
  rebuild_pairs(sm_lo, sm_hi, u, m, bw, x, out);
}

// ---- score product of one compressed K tile: sc += K . Q^T.  dump (debug instantiation only): where token 0 of this tile goes in the
// [token][128] dump of the head; rows >= nvalid are left alone.
template <bool WIN, bool DUMP>
__device__ __forceinline__ void k_decode(float* sc, const SideView& s, u32 area, const AttnView& w, int lane, const QFrag& Q, uint16_t* dump, int nvalid) {
  const int j = lane & 3, r = lane >> 2;
  u32 seg[2][2], pos[2] = {0u, 0u};                    // staged: the words of the lane's two segments;  not staged: tag bytes and positions
#pragma unroll
  for (int o = 0; o < 2; o++) {
    const u32x2 v = lds_u64(area + SEG_K + 256u * o + 8u * lane);
    seg[o][0] = WIN ? v.x : v.x & 0xFFu; seg[o][1] = v.y; pos[o] = v.x >> 16;
  }
  uint4 s0[2], s1[2]; u32 cd[2][3];
  float s2[4] = {0.f, 0.f, 0.f, 0.f};                  // second accumulator: two dependent MMA chains of four instead of one of eight
#pragma unroll
  for (int o = 0; o < 2; o++) {
    const uint8_t* m = s.sm + o * 1024 + 32 * lane;
    s0[o] = *reinterpret_cast<const uint4*>(m); s1[o] = *reinterpret_cast<const uint4*>(m + 16);
    const u32* c = reinterpret_cast<const u32*>(s.cd + o * 384 + 12 * lane);
    cd[o][0] = c[0]; cd[o][1] = c[1]; cd[o][2] = c[2];
  }
#pragma unroll
  for (int g = 0; g < 4; g++) {
    const u32x4 bw = lds_u128(w.bases + 80 * j + 16 * g);
    u32 f[2][4];
#pragma unroll
    for (int o = 0; o < 2; o++) {
      const u32 smlo = g == 0 ? s0[o].x : g == 1 ? s0[o].z : g == 2 ? s1[o].x : s1[o].z;
      const u32 smhi = g == 0 ? s0[o].y : g == 1 ? s0[o].w : g == 2 ? s1[o].y : s1[o].w;
      const u32 u = g == 0 ? code_bytes<0>(cd[o]) : g == 1 ? code_bytes<3>(cd[o]) : g == 2 ? code_bytes<6>(cd[o]) : code_bytes<9>(cd[o]);
      if (WIN) { if (g & 1) decode_staged<1>(smlo, smhi, u, seg[o][g >> 1], w, bw, f[o]); else decode_staged<0>(smlo, smhi, u, seg[o][g >> 1], w, bw, f[o]); }
      else decode_plain(smlo, smhi, u, seg[o][0] >> (2 * g), pos[o], s.glob, w, bw, f[o]);
    }
    if (DUMP) {
#pragma unroll
      for (int o = 0; o < 2; o++)
        if (8 * o + r < nvalid) {
          uint16_t* row = dump + (8 * o + r) * D + 32 * g + 2 * j;
#pragma unroll
          for (int i = 0; i < 4; i++) { uint16_t* e = row + (i & 1) + 8 * (i >> 1); e[0] = (uint16_t)(f[o][i] & 0xFFFFu); e[16] = (uint16_t)(f[o][i] >> 16); }
        }
    }
    mma16816(sc, f[0][0], f[1][0], f[0][1], f[1][1], Q.qa[2 * g][0], Q.qa[2 * g][1]);
    mma16816(s2, f[0][2], f[1][2], f[0][3], f[1][3], Q.qa[2 * g + 1][0], Q.qa[2 * g + 1][1]);
  }
  sc[0] += s2[0]; sc[1] += s2[1]; sc[2] += s2[2]; sc[3] += s2[3];
}
template <bool DUMP>
__device__ __forceinline__ void k_tile(float* sc, const SideView& s, int win, u32 area, const AttnView& w, int lane, const QFrag& Q, uint16_t* dump, int nvalid) {
  if (win & 1) k_decode<true, DUMP>(sc, s, area, w, lane, Q, dump, nvalid);
  else k_decode<false, DUMP>(sc, s, area, w, lane, Q, dump, nvalid);
}

// ---- value product of one compressed V tile
template <bool WIN, bool DUMP, int NSET>
__device__ __forceinline__ void v_decode(WarpAcc<NSET>& A, const SideView& s, u32 area, const AttnView& w, int lane, const PFrag<NSET>& P, uint16_t* dump, int nvalid) {
  const int j = lane & 3, r = lane >> 2;
  u32 seg[4], pos[4] = {0u, 0u, 0u, 0u};               // staged: the words of the lane's two groups of each token;  not staged: their tags and the position
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const u32 row = area + SEG_V + 32u * slot_token(j, i);
    if (WIN) seg[i] = lds_u32(row + 4u * r);
    else {
      const u32 v = lds_u32(row + 8u * (r >> 1)), tg = v & 0xFFu;
      seg[i] = r & 1 ? tg >> 4 : tg; pos[i] = (v >> 16) + (r & 1 ? seg_esc(tg & 15u) : 0u);
    }
  }
  const int swap = j >> 1;
  uint4 sm[4]; u32 cd[6];
#pragma unroll
  for (int i = 0; i < 4; i++) sm[i] = *reinterpret_cast<const uint4*>(s.sm + 64 * lane + 16 * (i & 1) + 32 * ((i >> 1) ^ swap));
#pragma unroll
  for (int i = 0; i < 6; i++) cd[i] = *reinterpret_cast<const u32*>(s.cd + 24 * lane + 4 * (i % 3) + 12 * ((i / 3) ^ swap));
#pragma unroll
  for (int g = 0; g < 2; g++) {
    const u32x4 bw = lds_u128(w.bases + PAIR_BASES_V + 32 * r + 16 * g);
    u32 f[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const u32 lo = g ? sm[i].z : sm[i].x, hi = g ? sm[i].w : sm[i].y;
      const u32 u = i == 0 ? (g ? code_bytes<3>(cd) : code_bytes<0>(cd)) : i == 1 ? (g ? code_bytes<9>(cd) : code_bytes<6>(cd)) :
                    i == 2 ? (g ? code_bytes<15>(cd) : code_bytes<12>(cd)) : (g ? code_bytes<21>(cd) : code_bytes<18>(cd));
      if (WIN) { if (g) decode_staged<1>(lo, hi, u, seg[i], w, bw, f[i]); else decode_staged<0>(lo, hi, u, seg[i], w, bw, f[i]); }
      else decode_plain(lo, hi, u, seg[i] >> (2 * g), pos[i], s.glob, w, bw, f[i]);
    }
    if (DUMP) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int tok = slot_token(j, i);
        if (tok < nvalid) {
#pragma unroll
          for (int q = 0; q < 4; q++) {                // word q = stored positions 16r + 8g + q, + 4  <->  channels 8(8g + q) + r, 8(8g + q + 4) + r
            dump[tok * D + 8 * (8 * g + q) + r] = (uint16_t)(f[i][q] & 0xFFFFu);
            dump[tok * D + 8 * (8 * g + q + 4) + r] = (uint16_t)(f[i][q] >> 16);
          }
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const u32 w0[4] = {f[0][2 * h], f[1][2 * h], f[2][2 * h], f[3][2 * h]};
      const u32 w1[4] = {f[0][2 * h + 1], f[1][2 * h + 1], f[2][2 * h + 1], f[3][2 * h + 1]};
      pv_words(A, 2 * g + h, w0, w1, P);
    }
  }
}
template <bool DUMP, int NSET>
__device__ __forceinline__ void v_tile(WarpAcc<NSET>& A, const SideView& s, int win, u32 area, const AttnView& w, int lane, const PFrag<NSET>& P, uint16_t* dump, int nvalid) {
  if (win & 2) v_decode<true, DUMP, NSET>(A, s, area, w, lane, P, dump, nvalid);
  else v_decode<false, DUMP, NSET>(A, s, area, w, lane, P, dump, nvalid);
}

// ---- raw BF16 tiles [16][128] in global memory (rows >= nvalid are not read): the slot layout's tail, the paged layout's filling block
// and its tiles that stayed raw
template <bool DUMP>
__device__ __forceinline__ void raw_scores(float* sc, const uint16_t* kraw, int nvalid, int lane, const QFrag& Q, uint16_t* dump) {
  const int j = lane & 3, r = lane >> 2;
#pragma unroll
  for (int s = 0; s < 8; s++) {
    u32 x[2][2];                                       // [row half][16 channels on]
#pragma unroll
    for (int o = 0; o < 2; o++) {
      const int at = (8 * o + r) * D + 32 * (s >> 1) + 2 * j + 8 * (s & 1);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        x[o][i] = 8 * o + r < nvalid ? *reinterpret_cast<const u32*>(kraw + at + 16 * i) : 0u;
        if (DUMP && 8 * o + r < nvalid) *reinterpret_cast<u32*>(dump + at + 16 * i) = x[o][i];
      }
    }
    mma16816(sc, prmt(x[0][0], x[0][1], 0x5410), prmt(x[1][0], x[1][1], 0x5410), prmt(x[0][0], x[0][1], 0x7632), prmt(x[1][0], x[1][1], 0x7632), Q.qa[s][0], Q.qa[s][1]);
  }
}
template <bool DUMP, int NSET>
__device__ __forceinline__ void raw_accum(WarpAcc<NSET>& A, const uint16_t* vraw, int nvalid, int lane, const PFrag<NSET>& P, uint16_t* dump) {
  const int j = lane & 3, r = lane >> 2;
#pragma unroll
  for (int mt = 0; mt < 4; mt++) {
    u32 w0[4], w1[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int tok = slot_token(j, t);
      const bool ok = tok < nvalid;
      u32 e[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const int at = tok * D + 8 * acc_channel(mt, c) + r;
        e[c] = ok ? vraw[at] : 0u;
        if (DUMP && ok) dump[at] = (uint16_t)e[c];
      }
      w0[t] = e[0] | (e[1] << 16); w1[t] = e[2] | (e[3] << 16);
    }
    pv_words(A, mt, w0, w1, P);
  }
}

// ---- one element of a tile, read from global memory bit by bit (sum_exact): where the storage order puts it, its code, its group's tag and escape
// bytes.  tags, esc_at: tag word of the token's row and position of the row's first escape byte inside the tile.
struct PlainSide { const uint8_t *sm, *cd, *esc, *b3, *b4; const uint16_t* raw; };         // raw: the tile as BF16 rows, then nothing else is read
template <bool VSIDE> __device__ __forceinline__ float plain_element(const PlainSide& s, int tok, int ch, u32 tags, int esc_at) {
  if (s.raw) return __uint_as_float((u32)s.raw[tok * D + ch] << 16);
  int group, k, sm_at, cd_at;                        // group of the row, element inside it, byte of the sign/mantissa, bit of the code
  if (VSIDE) {
    const int r = ch & 7, n = ch >> 3, lane = 4 * r + ((tok & 7) >> 1), t = (tok & 1) + 2 * (tok >> 3);
    group = 2 * r + (n >> 3); k = n & 7; sm_at = 64 * lane + 16 * t + n; cd_at = 8 * (24 * lane + 6 * t) + 3 * n;
  } else {
    const int j = (ch & 7) >> 1, at = 4 * (ch >> 4) + (ch & 1) + 2 * ((ch >> 3) & 1), lane = 4 * (tok & 7) + j, o = tok >> 3;
    group = 4 * j + (at >> 3); k = at & 7; sm_at = 1024 * o + 32 * lane + at; cd_at = 8 * (384 * o + 12 * lane) + 3 * at;
  }
  const u32 sm = s.sm[sm_at], two = (u32)s.cd[cd_at >> 3] | ((cd_at & 7) > 5 ? (u32)s.cd[(cd_at >> 3) + 1] << 8 : 0u), code = (two >> (cd_at & 7)) & 7u, tag = (tags >> (2 * group)) & 3u;
  const uint8_t* esc = s.esc + esc_at + esc_prefix(tags, 2 * group);
  u32 e = s.b3[ch] + code;
  if (tag == 1u) e = s.b4[ch] + code + (((u32)esc[0] >> k) & 1u) * 8u;
  if (tag == 3u) { const int bit = 5 * k; e = code | (((((u32)esc[bit >> 3] | ((bit & 7) > 3 ? (u32)esc[(bit >> 3) + 1] << 8 : 0u)) >> (bit & 7)) & 31u) << 3); }
  return __uint_as_float(((sm & 0x80u) << 24) | ((e & 0xFFu) << 23) | ((sm & 0x7Fu) << 16));
}

}  // namespace gaac
