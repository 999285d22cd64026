// Warp-level pieces of the fused decode attention: asynchronous copies, the rebuild of a compressed 16-token tile into tensor-core
// fragments, the score and value products and the online softmax step.  Used by the kernels of gaac_attn.cu.
//
// What bounds them: instruction issue and the integer (ALU) pipe, whose rate is half the issue rate, not HBM.  Measured on a B200
// at batch 1, 32 query / 8 kv heads, 65536 tokens: 1354 warp instructions per (K tile + V tile) at 67 % issue slots used before the
// forms below, of which the group decoder itself is about 530; the rest was copy issue per warp, escape offsets through two
// lookups per row, a transpose of the V fragments and softmax work for padding heads.
//
// Head columns.  The tensor-core tile has 8 columns.  Query heads are handled in sets of four (NSET = 1 for a GQA group of up to
// 4, 2 for 5..8); lane j of a quad works for head 4 * set + j throughout:
//   scores  S^T[16 tok x 8] = K[16 x 128] . Q^T : column 2j = head j of set 0, column 2j + 1 = head j of set 1 (zero without it)
//   values, one set: a rebuilt word holds TWO channels of one token, so O^T += V^T . P^T contracts over (token, channel parity) and column
//           2j + parity takes (P, 0) or (0, P): the words go into the product as they were decoded, with no transpose, and each lane
//           gets both channels of its own head.  16 products per tile, as many as a transposed form has for 8 heads
//   values, two sets: the columns are the heads, as for the scores, and the words of two tokens are transposed by 32 byte permutes per tile.  The form
//           above takes 32 products and 16 registers of weights where this takes 16 and 4, and was slower: group of 8, 8 kv heads, 65536
//           tokens 67.1 us, now 64.4; paged 32768 40.1 -> 38.7; head_dim 256, 8 x 8000: 119 -> 111
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
__device__ __forceinline__ void mbar_add_tx(u32 mbar, u32 bytes) { asm volatile("mbarrier.expect_tx.shared::cta.b64 [%0], %1;\n" ::"r"(mbar), "r"(bytes) : "memory"); }
__device__ __forceinline__ void bulk_g2s(u32 dst, const void* src, u32 bytes, u32 mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
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
// The same for a count in shared memory that other warps raise: waits until it is at least `least`.
__device__ __forceinline__ bool wait_count(u32 addr, int least) {
  for (int it = 0; it < MBAR_WAIT_LIMIT; it++) {
    int v;
    asm volatile("ld.relaxed.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    if (v >= least) return true;
  }
  return false;
}
__device__ __forceinline__ float fast_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// What a warp needs to know of a tile besides its staged bytes.  Slot layout: offsets of the tile's escape bytes inside the head's
// escape bytes.  Paged layout: the mode-table entries (>= 0: compressed slot, < 0: bit-complement of a raw tile of the pool).
struct TileMeta { int mk, mv; };

// ---- running state of one warp.  acc[set][mt][c] = O[head 4 * set + j][channel 8 * (4 * mt + c) + r]; m, l in the exp2 domain, l summed over
// this lane's tokens only
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

// Q^T B-fragments of the score product.  Lane (j, r) provides column r = head 4 * (r & 1) + (r >> 1): for k-step s the words
// q[16s + 2j, +1] and q[16s + 2j + 8, +9] of that head (zero where the group has no such head).
struct QFrag { u32 qa[8][2]; };
__device__ __forceinline__ int q_head(int r) { return 4 * (r & 1) + (r >> 1); }
__device__ __forceinline__ void load_q(QFrag& Q, const uint16_t* q0, long head_stride, int G, int lane) {
  const int j = lane & 3, h = q_head(lane >> 2);
  const uint16_t* qp = q0 + (h < G ? h : 0) * head_stride;
#pragma unroll
  for (int s = 0; s < 8; s++) {
    Q.qa[s][0] = h < G ? *reinterpret_cast<const u32*>(qp + 16 * s + 2 * j) : 0u;
    Q.qa[s][1] = h < G ? *reinterpret_cast<const u32*>(qp + 16 * s + 2 * j + 8) : 0u;
  }
}

// Weights of one tile as B-fragments of the value product.  A weight enters as the sum of two BF16 numbers, its rounded value (hi) and the rounded
// remainder (lo), which brings its relative error to 2^-16.  One set: [0]: tokens 2j (b0) and 2j + 1 (b1), [1]: tokens 2j + 8 and 2j + 9.  Two: [0]:
// tokens 2j, 2j + 1, [1]: tokens 2j + 8, 2j + 9.
template <int NSET> struct PFrag;
template <> struct PFrag<1> { u32 hi[2][2], lo[2][2]; };
template <> struct PFrag<2> { u32 hi[2], lo[2]; };
__device__ __forceinline__ u32 pack_bf16(float lo, float hi) { __nv_bfloat162 x = __floats2bfloat162_rn(lo, hi); return *reinterpret_cast<u32*>(&x); }
// what the rounding of a pair dropped, which fp32 holds exactly, rounded in turn
__device__ __forceinline__ u32 pack_rest(float lo, float hi, u32 rounded) { return pack_bf16(lo - __uint_as_float(rounded << 16), hi - __uint_as_float(rounded & 0xFFFF0000u)); }

// p0, p8: this lane's weights of tokens r and r + 8 for head j of each set.
// One set: as column r of the value product the lane needs those of head r >> 1 for tokens 2j, 2j + 1, 2j + 8, 2j + 9, in the low (parity 0) or high
// (parity 1) half of a word whose other half is zero.
__device__ __forceinline__ void put_weights(PFrag<1>& P, const float (&p0)[1], const float (&p8)[1], int lane) {
  const int j = lane & 3, r = lane >> 2, src = 8 * j + (r >> 1);
  const u32 sel0 = (r & 1) ? 0x1044u : 0x4410u, sel8 = (r & 1) ? 0x3244u : 0x4432u;
  const u32 H = pack_bf16(p0[0], p8[0]), L = pack_rest(p0[0], p8[0], H);
  const u32 ha = __shfl_sync(FULLM, H, src), hb = __shfl_sync(FULLM, H, src + 4), la = __shfl_sync(FULLM, L, src), lb = __shfl_sync(FULLM, L, src + 4);
  P.hi[0][0] = prmt(ha, 0u, sel0); P.hi[0][1] = prmt(hb, 0u, sel0); P.hi[1][0] = prmt(ha, 0u, sel8); P.hi[1][1] = prmt(hb, 0u, sel8);
  P.lo[0][0] = prmt(la, 0u, sel0); P.lo[0][1] = prmt(lb, 0u, sel0); P.lo[1][0] = prmt(la, 0u, sel8); P.lo[1][1] = prmt(lb, 0u, sel8);
}
// Two: column r is head r >> 1 of set r & 1, its words hold two tokens.
__device__ __forceinline__ void put_weights(PFrag<2>& P, const float (&p0)[2], const float (&p8)[2], int lane) {
  const int j = lane & 3, r = lane >> 2, src = 8 * j + (r >> 1);
  const u32 sel = (r & 1) ? 0x7632u : 0x5410u;
  const u32 h0 = pack_bf16(p0[0], p0[1]), h8 = pack_bf16(p8[0], p8[1]), l0 = pack_rest(p0[0], p0[1], h0), l8 = pack_rest(p8[0], p8[1], h8);
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

// Value product of words i, i + 1 (i = 2 * mt) of the lane's four tokens (2j, 2j + 1, 2j + 8, 2j + 9).
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
constexpr int PATCH_MAX = 64;                               // raw groups of a tile (K and V together) that the patch table holds
constexpr int PATCH_BYTES = PATCH_MAX * 8, WALK_BYTES = 32 * 16;
constexpr int WARP_SCRATCH = PATCH_BYTES + WALK_BYTES;      // shared memory of a warp besides its stages: patch table, segment positions per lane

// One side (K or V) of a staged tile.  esc = shared-memory address of its first escape byte, glob = the same bytes in global memory, avail = staged escape
// bytes.
struct SideView { const uint8_t *sm, *cd, *fl; u32 esc; const uint8_t* glob; int avail; };
// ---- where a lane's escape bytes are.  A lane owns 8 groups of a K tile (tokens r and r + 8, groups 4j .. 4j + 3 of each) and 8 of a V tile
// (groups 2r, 2r + 1 of tokens 2j, 2j + 1, 2j + 8, 2j + 9).
//   tags  2 bits per group: K segments (8 bits) at bits 0 and 8, V segments (4 bits) at bits 16, 20, 24, 28
//   k, v  position of each segment's first escape byte inside the tile side, two per word
//   win   bit 0 / 1: the K / V side takes the decoder with staged escape bytes
struct TilePlan { u32 tags, k, v[2]; int win; };

// Turn the raw-tier groups of a staged tile (K and V in one pass) into patch-table entries, so that the group decoder needs no branch.  A lane
// walks its own raw groups: read the five payload bytes, spread the 5-bit fields to byte positions, take off the 4-bit-window base words (the
// decoder adds them to every promoted group), store the two words as entry k, and write k over the first payload byte, which is where the
// decoder looks.  Returns false when there are more than PATCH_MAX (the caller then takes the decoder that reads global memory, so the bytes
// written over do not matter).  At a raw share of 0.75 % a tile pair has 3.8 raw groups, hardly ever two in one lane: one trip.
__device__ __forceinline__ bool build_raw_patches(u32 raw_bits, const TilePlan& t, u32 esc_k, u32 esc_v, const WarpView& w, int lane) {
  u32 some = __ballot_sync(FULLM, raw_bits != 0u);
  if (!some) return true;
  const u32 mine = w.scratch + PATCH_BYTES + 16 * lane, j = lane & 3, r = lane >> 2;
  sts_u128(mine, prmt(t.k, 0u, 0x1010), prmt(t.k, 0u, 0x3232), t.v[0], t.v[1]);        // position by quarter of the tag word: the walk picks one at run time
  u32 base = 0;
  do {
    const u32 n = base + (u32)popc(some);
    if (n > PATCH_MAX) return false;
    if (raw_bits) {
      const u32 bit = (u32)__ffs((int)raw_bits) - 1u;                // upper tag bit of the group
      raw_bits &= raw_bits - 1u;
      const bool isv = bit >= 16u;
      const u32 first = bit & (isv ? ~3u : ~7u);                     // first tag bit of its segment
      const u32 below = (t.tags >> first) & ((1u << (bit - 1u - first)) - 1u);
      const u32 pl = (isv ? esc_v : esc_k) + lds_u16(mine + ((bit >> 2) << 1)) + seg_esc(below);
      const u32 k = base + (u32)popc(some & ((1u << lane) - 1u));
      const u32x4 bw = lds_u128(w.bases + (isv ? BASES_V + 32u * r + 8u * (bit & 2u) : 64u * j + 8u * (bit & 6u)));
      const u32x2 x = raw_addends(lds_u32(pl & ~3u), lds_u32((pl & ~3u) + 4u), 8u * (pl & 3u), bw.x + bw.z, bw.y + bw.w);
      sts_u64(w.scratch + 8u * k, x.x, x.y);
      sts_u8(pl, k);
    }
    base = n;
    some = __ballot_sync(FULLM, raw_bits != 0u);
  } while (some);
  __syncwarp();
  return true;
}

__device__ __forceinline__ TilePlan plan_tile(const SideView& ks, const SideView& vs, bool rawk, bool rawv, const WarpView& w, int lane) {
  const int j = lane & 3, r = lane >> 2;
  TilePlan t;
  u32 k0 = 0, k1 = 0, v0 = 0, v1 = 0, v2 = 0, v3 = 0;
  if (!rawk) { k0 = ks.fl[lane]; k1 = ks.fl[32 + lane]; }                                     // byte j of row r's tag word is byte `lane` of the octet's 32
  if (!rawv) {
    const uint2 a = *reinterpret_cast<const uint2*>(vs.fl + 8 * j), b = *reinterpret_cast<const uint2*>(vs.fl + 32 + 8 * j);      // tag words of the four tokens
    v0 = (a.x >> (4 * r)) & 15u; v1 = (a.y >> (4 * r)) & 15u; v2 = (b.x >> (4 * r)) & 15u; v3 = (b.y >> (4 * r)) & 15u;
  }
  u32 ktot, vtot;
  tile_positions<true, true>(k0, k1, v0, v1, v2, v3, j, t.k, ktot, t.v, vtot);
  t.tags = mad_k<256u>(k1, k0) + mad_k<65536u>(v0, mad_k<1048576u>(v1, mad_k<16777216u>(v2, mad_k<268435456u>(v3, 0u))));
  const int total_k = (int)((ktot & 0xFFFFu) + (ktot >> 16)), total_v = (int)((vtot & 0xFFFFu) + (vtot >> 16));
  t.win = (total_k <= ks.avail ? 1 : 0) | (total_v <= vs.avail ? 2 : 0);
  const u32 sides = ((t.win & 1) ? 0xAAAAu : 0u) | ((t.win & 2) ? 0xAAAA0000u : 0u);
  if (!build_raw_patches(t.tags & sides, t, ks.esc, vs.esc, w, lane)) t.win = 0;
  return t;
}

// ---- score product of one compressed K tile: sc += K . Q^T.  dump (debug instantiation only): where token 0 of this tile goes in the
// [token][128] dump of the head; rows >= nvalid are left alone.
template <bool WIN, bool DUMP>
__device__ __forceinline__ void k_decode(float* sc, const SideView& s, const TilePlan& t, const WarpView& w, int lane, const QFrag& Q, uint16_t* dump, int nvalid) {
  const int j = lane & 3, r = lane >> 2;
  const u32 from = WIN ? s.esc - w.zero : 0u;
  u32 pos[2] = {(t.k & 0xFFFFu) + from, (t.k >> 16) + from};
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
    const u32x4 bw = lds_u128(w.bases + 64 * j + 16 * g);
    u32 f[2][4];
#pragma unroll
    for (int o = 0; o < 2; o++) {
      const u32 smlo = g == 0 ? s0[o].x : g == 1 ? s0[o].z : g == 2 ? s1[o].x : s1[o].z;
      const u32 smhi = g == 0 ? s0[o].y : g == 1 ? s0[o].w : g == 2 ? s1[o].y : s1[o].w;
      const u32 z = g == 0 ? group_codes<0>(cd[o]) : g == 1 ? group_codes<3>(cd[o]) : g == 2 ? group_codes<6>(cd[o]) : group_codes<9>(cd[o]);
      decode_group_dev<WIN>(smlo, smhi, z, t.tags >> (8 * o + 2 * g), pos[o], s.glob, w, bw, f[o]);
    }
    if (DUMP) {
#pragma unroll
      for (int o = 0; o < 2; o++)
        if (8 * o + r < nvalid) {
          u32* row = reinterpret_cast<u32*>(dump + (8 * o + r) * D);
          row[(32 * g + 2 * j) >> 1] = f[o][0]; row[(32 * g + 2 * j + 8) >> 1] = f[o][1];
          row[(32 * g + 16 + 2 * j) >> 1] = f[o][2]; row[(32 * g + 16 + 2 * j + 8) >> 1] = f[o][3];
        }
    }
    mma16816(sc, f[0][0], f[1][0], f[0][1], f[1][1], Q.qa[2 * g][0], Q.qa[2 * g][1]);
    mma16816(s2, f[0][2], f[1][2], f[0][3], f[1][3], Q.qa[2 * g + 1][0], Q.qa[2 * g + 1][1]);
  }
  sc[0] += s2[0]; sc[1] += s2[1]; sc[2] += s2[2]; sc[3] += s2[3];
}
template <bool DUMP>
__device__ __forceinline__ void k_tile(float* sc, const SideView& s, const TilePlan& t, const WarpView& w, int lane, const QFrag& Q, uint16_t* dump, int nvalid) {
  if (t.win & 1) k_decode<true, DUMP>(sc, s, t, w, lane, Q, dump, nvalid);
  else k_decode<false, DUMP>(sc, s, t, w, lane, Q, dump, nvalid);
}

// ---- value product of one compressed V tile
template <bool WIN, bool DUMP, int NSET>
__device__ __forceinline__ void v_decode(WarpAcc<NSET>& A, const SideView& s, const TilePlan& t, const WarpView& w, int lane, const PFrag<NSET>& P, uint16_t* dump, int nvalid) {
  const int j = lane & 3, r = lane >> 2;
  const u32 from = WIN ? s.esc - w.zero : 0u;
  u32 pos[4] = {(t.v[0] & 0xFFFFu) + from, (t.v[0] >> 16) + from, (t.v[1] & 0xFFFFu) + from, (t.v[1] >> 16) + from};
  uint4 sm[4]; u32 cd[6];
#pragma unroll
  for (int i = 0; i < 4; i++) sm[i] = *reinterpret_cast<const uint4*>(s.sm + 64 * lane + 16 * i);
  {
    const uint2* c2 = reinterpret_cast<const uint2*>(s.cd + 24 * lane);
    const uint2 ca = c2[0], cb = c2[1], cc = c2[2];
    cd[0] = ca.x; cd[1] = ca.y; cd[2] = cb.x; cd[3] = cb.y; cd[4] = cc.x; cd[5] = cc.y;
  }
#pragma unroll
  for (int g = 0; g < 2; g++) {
    const u32x4 bw = lds_u128(w.bases + BASES_V + 32 * r + 16 * g);
    u32 f[4][4];
    decode_group_dev<WIN>(g ? sm[0].z : sm[0].x, g ? sm[0].w : sm[0].y, g ? group_codes<3>(cd) : group_codes<0>(cd), t.tags >> (16 + 2 * g), pos[0], s.glob, w, bw, f[0]);
    decode_group_dev<WIN>(g ? sm[1].z : sm[1].x, g ? sm[1].w : sm[1].y, g ? group_codes<9>(cd) : group_codes<6>(cd), t.tags >> (20 + 2 * g), pos[1], s.glob, w, bw, f[1]);
    decode_group_dev<WIN>(g ? sm[2].z : sm[2].x, g ? sm[2].w : sm[2].y, g ? group_codes<15>(cd) : group_codes<12>(cd), t.tags >> (24 + 2 * g), pos[2], s.glob, w, bw, f[2]);
    decode_group_dev<WIN>(g ? sm[3].z : sm[3].x, g ? sm[3].w : sm[3].y, g ? group_codes<21>(cd) : group_codes<18>(cd), t.tags >> (28 + 2 * g), pos[3], s.glob, w, bw, f[3]);
    if (DUMP) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int tok = 2 * j + (i & 1) + 8 * (i >> 1);
        if (tok < nvalid) {
#pragma unroll
          for (int q = 0; q < 4; q++) {                // word q = stored positions 16r + 8g + 2q, +1  <->  channels 8(8g + 2q) + r, 8(8g + 2q + 1) + r
            dump[tok * D + 8 * (8 * g + 2 * q) + r] = (uint16_t)(f[i][q] & 0xFFFFu);
            dump[tok * D + 8 * (8 * g + 2 * q + 1) + r] = (uint16_t)(f[i][q] >> 16);
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
__device__ __forceinline__ void v_tile(WarpAcc<NSET>& A, const SideView& s, const TilePlan& t, const WarpView& w, int lane, const PFrag<NSET>& P, uint16_t* dump, int nvalid) {
  if (t.win & 2) v_decode<true, DUMP, NSET>(A, s, t, w, lane, P, dump, nvalid);
  else v_decode<false, DUMP, NSET>(A, s, t, w, lane, P, dump, nvalid);
}

// ---- raw BF16 tiles [16][128] in global memory (rows >= nvalid are not read): the slot layout's tail, the paged layout's filling block
// and its tiles that stayed raw
template <bool DUMP>
__device__ __forceinline__ void raw_scores(float* sc, const uint16_t* kraw, int nvalid, int lane, const QFrag& Q, uint16_t* dump) {
  const int j = lane & 3, r = lane >> 2;
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const uint16_t* k0 = kraw + r * D + 16 * s + 2 * j;
    const uint16_t* k8 = k0 + 8 * D;
    const u32 a0 = r < nvalid ? *reinterpret_cast<const u32*>(k0) : 0u, a2 = r < nvalid ? *reinterpret_cast<const u32*>(k0 + 8) : 0u;
    const u32 a1 = r + 8 < nvalid ? *reinterpret_cast<const u32*>(k8) : 0u, a3 = r + 8 < nvalid ? *reinterpret_cast<const u32*>(k8 + 8) : 0u;
    if (DUMP) {
      if (r < nvalid) { u32* row = reinterpret_cast<u32*>(dump + r * D); row[(16 * s + 2 * j) >> 1] = a0; row[(16 * s + 2 * j + 8) >> 1] = a2; }
      if (r + 8 < nvalid) { u32* row = reinterpret_cast<u32*>(dump + (r + 8) * D); row[(16 * s + 2 * j) >> 1] = a1; row[(16 * s + 2 * j + 8) >> 1] = a3; }
    }
    mma16816(sc, a0, a1, a2, a3, Q.qa[s][0], Q.qa[s][1]);
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
      const int tok = 2 * j + (t & 1) + 8 * (t >> 1);
      const uint16_t* vr = vraw + tok * D + 8 * (4 * mt) + r;
      const bool ok = tok < nvalid;
      const u32 e0 = ok ? vr[0] : 0u, e1 = ok ? vr[8] : 0u, e2 = ok ? vr[16] : 0u, e3 = ok ? vr[24] : 0u;
      w0[t] = e0 | (e1 << 16); w1[t] = e2 | (e3 << 16);
      if (DUMP && ok) {
        uint16_t* o = dump + tok * D + 8 * (4 * mt) + r;
        o[0] = (uint16_t)e0; o[8] = (uint16_t)e1; o[16] = (uint16_t)e2; o[24] = (uint16_t)e3;
      }
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
