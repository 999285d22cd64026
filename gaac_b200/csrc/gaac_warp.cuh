// Warp-level tile encode / decode built on the lane-level functions of gaac_tile.h.
// One warp owns one 16-token tile.  Shared by the page encoder, the slot-cache append and the paged store kernels.
#pragma once
#include <cuda_runtime.h>
#include "gaac_lane.cuh"

namespace gaac {

constexpr int XS_STRIDE = 136;                      // u16 per staged row: 272 B keeps 16-byte alignment and spreads banks
constexpr unsigned FULL = 0xffffffffu;

// Per-warp scratch in shared memory.
struct WarpScratch {
  uint16_t xs[T * XS_STRIDE];                        // staged tile, natural channel order
};
// A decoder's scratch: behind the rows room for the `most` escape bytes that a tile may have, from the 4-byte boundary at or below the first.  What follows them may be read: a
// segment's four raw groups, and a word.
__host__ __device__ constexpr int decode_scratch_bytes(int most) { return (int)sizeof(WarpScratch) + ((most + 3 + 20 + 8 + 15) & ~15); }
// What the warps of a CTA that decodes tiles of one (kind, head) share: the base words.
struct DecodeTables {
  __align__(16) uint8_t bases[BASES_BYTES];
};

// Encoded tile held in registers, one lane's share.  8 groups per lane for both kinds, in runs of consecutive groups of one row (segments):
//   K: idx = 4*o + g  -> row 8o + (lane>>2), group 4*(lane&3) + g          V: idx = 2*t + g -> row tok(t), group 2*(lane>>2) + g
struct LaneTile {
  u32 sm[16];        // K: [o][8] words;  V: [t][4] words
  u32 cd[6];         // K: [o][3] words;  V: 192 code bits (4 token slots x 48)
  u32 esc1[8];       // the escape byte of a tier 1 group
  u32 tags;          // 2 bits per idx
  u32 pos[2];        // where the segments' escape bytes begin inside the tile: K: pos[0] = {octet 0, octet 1};  V: pos[t >> 1] = {t & ~1, t | 1} (16 bits each)
};

__device__ __forceinline__ int v_tok(int j, int t) { return 2 * j + (t & 1) + 8 * (t >> 1); }
// Stage rows [row0, row0+16) of a [*, 128] bf16 matrix into ws.xs; rows >= nvalid are zero-filled.
__device__ __forceinline__ void stage_rows(WarpScratch& ws, const uint16_t* src, long row_stride, int nvalid, int lane) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    int c = lane + 32 * k, row = c >> 4, col = (c & 15) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (row < nvalid) v = *reinterpret_cast<const uint4*>(src + (long)row * row_stride + col);
    *reinterpret_cast<uint4*>(&ws.xs[row * XS_STRIDE + col]) = v;
  }
}

// The same staging with asynchronous 16-byte copies (rows >= nvalid are zero-filled by the copy unit): the caller commits the
// group and waits for it before encode_tile_warp, so the rows of the next tile travel while the current one is encoded.
__device__ __forceinline__ void stage_rows_async(WarpScratch& ws, const uint16_t* src, long row_stride, int nvalid, int lane) {
  // piece k of a lane: row 2k + (lane >> 4), columns 8 * (lane & 15) .. +7: one source and one destination address per lane, a
  // fixed step per piece
  const int r0 = lane >> 4, col = (lane & 15) * 8;
  const uint16_t* g = src + (long)r0 * row_stride + col;
  const unsigned d = (unsigned)__cvta_generic_to_shared(&ws.xs[r0 * XS_STRIDE + col]);
  const long step = 2 * row_stride;
  if (nvalid == T) {
#pragma unroll
    for (int k = 0; k < 8; k++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + k * (2 * XS_STRIDE * 2)), "l"(g + k * step) : "memory");
  } else {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const bool live = 2 * k + r0 < nvalid;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d + k * (2 * XS_STRIDE * 2)), "l"(live ? g + k * step : src), "r"(live ? 16 : 0) : "memory");
    }
  }
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Four 8 x 8 matrices of 16-bit values out of the staged tile: channels 16s .. 16s + 7 and 16s + 8 .. 16s + 15 of tokens 0..7 (w[0], w[1]) and of
// tokens 8..15 (w[2], w[3]).  `at`: the lane's row address, &xs[(8 * (lane >> 4) + (lane & 7)) * XS_STRIDE + 8 * ((lane >> 3) & 1)].  Rows are 68
// words apart, so the eight rows of a matrix lie in different banks.
//   plain:      lane (j, r) gets channels 2j, 2j + 1 of token r, which is how a lane owns a K tile
//   transposed: lane (j, r) gets channel r of tokens 2j, 2j + 1, which is how it owns a V tile
template <bool TRANS> __device__ __forceinline__ void load_matrices(u32 (&w)[4], u32 at, int s) {
  if (!TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(at + 32 * s) : "memory");
  else asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(at + 32 * s) : "memory");
}
__device__ __forceinline__ u32 matrix_row_address(const WarpScratch& ws, int lane) {
  return (u32)__cvta_generic_to_shared(&ws.xs[(8 * (lane >> 4) + (lane & 7)) * XS_STRIDE + 8 * ((lane >> 3) & 1)]);
}
// Encode the staged tile.  Rows >= nvalid become empty rows (sm = 0, codes = 0, tag word 0); they must have been staged as zeros.  On return
// every lane holds its share in `lt` and the tile's escape byte count is returned (same in all lanes).
// Bound by instruction issue: 16-bit loads one by one, a byte-exact subtraction per window, a table of tags in shared memory and a branch per
// escape byte made 1205 warp instructions per tile; now the fragments come in by ldmatrix, a window is one subtraction per word and the
// positions of the escape bytes come from one warp scan.  [8, 65536, 128]: 60 (K) / 66 us (V) -> 39 / 41, that is 5.9 / 5.6 TB/s of input and output.
template <int KIND_V>
__device__ __forceinline__ int encode_tile_warp(WarpScratch& ws, int nvalid, const u32* b3w, const u32* b4w, int lane, LaneTile& lt) {
  const int j = lane & 3, r = lane >> 2;
  const u32 at = matrix_row_address(ws, lane);
  lt.tags = 0;
  __syncwarp();                                      // staged rows visible
  u32 c24[8];
#pragma unroll
  for (int g = 0; g < (KIND_V ? 2 : 4); g++) {
    if (!KIND_V) {
      u32 e[2][2];                                   // [octet][half group]
#pragma unroll
      for (int h = 0; h < 2; h++) {
        u32 w[4];
        load_matrices<false>(w, at, 2 * g + h);
        split_bf16x4(w[0], w[1], lt.sm[2 * g + h], e[0][h]);
        split_bf16x4(w[2], w[3], lt.sm[8 + 2 * g + h], e[1][h]);
      }
#pragma unroll
      for (int o = 0; o < 2; o++)
        lt.tags |= encode_group_codes(e[o][0], e[o][1], b3w[2 * g], b3w[2 * g + 1], b4w[2 * g], b4w[2 * g + 1], c24[4 * o + g], lt.esc1[4 * o + g]) << (8 * o + 2 * g);
    } else {
      u32 e[4][2];                                   // [token slot][half group]
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = 2 * g + h;                     // channels 32i .. 32i + 31: four matrices of each token half
        u32 a[4], b[4];
        load_matrices<true>(a, at, 2 * i); load_matrices<true>(b, at, 2 * i + 1);
#pragma unroll
        for (int th = 0; th < 2; th++) split_token_pairs(a[2 * th], a[2 * th + 1], b[2 * th], b[2 * th + 1], lt.sm[8 * th + i], e[2 * th][h], lt.sm[8 * th + 4 + i], e[2 * th + 1][h]);      // tokens 2j, 2j + 1 (+ 8)
      }
#pragma unroll
      for (int t = 0; t < 4; t++)
        lt.tags |= encode_group_codes(e[t][0], e[t][1], b3w[2 * g], b3w[2 * g + 1], b4w[2 * g], b4w[2 * g + 1], c24[2 * t + g], lt.esc1[2 * t + g]) << (4 * t + 2 * g);
    }
  }
  if (nvalid < T) {                                  // empty rows: zeros as values, which the windows above may have coded as anything
#pragma unroll
    for (int t = 0; t < (KIND_V ? 4 : 2); t++) {
      if ((KIND_V ? v_tok(j, t) : 8 * t + r) >= nvalid) {
        lt.tags &= KIND_V ? ~(0xFu << (4 * t)) : ~(0xFFu << (8 * t));
#pragma unroll
        for (int i = 0; i < (KIND_V ? 2 : 4); i++) c24[(KIND_V ? 2 : 4) * t + i] = 0u;
      }
    }
  }
  join_codes(c24[0], c24[1], c24[2], c24[3], lt.cd);
  join_codes(c24[4], c24[5], c24[6], c24[7], lt.cd + 3);
  u32 total, none;
  if (!KIND_V) tile_positions<true, false>(lt.tags & 0xFFu, lt.tags >> 8, 0u, 0u, 0u, 0u, j, lt.pos[0], total, lt.pos, none);
  else tile_positions<false, true>(0u, 0u, lt.tags & 15u, (lt.tags >> 4) & 15u, (lt.tags >> 8) & 15u, lt.tags >> 12, j, none, none, lt.pos, total);
  return (int)((total & 0xFFFFu) + (total >> 16));
}

// 32 bytes in one store (the address is a multiple of 32)
__device__ __forceinline__ void store_32(void* p, const u32* w) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
// Write one lane's sign/mantissa bytes, code bytes and tags of the tile (tile-relative destinations in global memory; fl_dst: 16 tag words).
// A lane's sign/mantissa bytes are 32 (K) or 64 (V) contiguous ones: whole sectors where the destination is 32-byte aligned, which only a
// paged slot whose stride is an odd multiple of 16 is not.
template <int KIND_V>
__device__ __forceinline__ void store_tile_payload(const LaneTile& lt, uint8_t* sm_dst, uint8_t* cd_dst, uint8_t* fl_dst, int lane) {
  constexpr int STEP = KIND_V ? 32 : 1024;
  uint8_t* s0 = sm_dst + (KIND_V ? 64 : 32) * lane;
  if ((reinterpret_cast<uintptr_t>(sm_dst) & 31) == 0) { store_32(s0, lt.sm); store_32(s0 + STEP, lt.sm + 8); }
  else {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint4* s = reinterpret_cast<uint4*>(s0 + h * STEP);
      s[0] = make_uint4(lt.sm[8 * h], lt.sm[8 * h + 1], lt.sm[8 * h + 2], lt.sm[8 * h + 3]);
      s[1] = make_uint4(lt.sm[8 * h + 4], lt.sm[8 * h + 5], lt.sm[8 * h + 6], lt.sm[8 * h + 7]);
    }
  }
  if (!KIND_V) {
#pragma unroll
    for (int o = 0; o < 2; o++) {
      u32* c = reinterpret_cast<u32*>(cd_dst + o * 384 + 12 * lane);
      c[0] = lt.cd[3 * o]; c[1] = lt.cd[3 * o + 1]; c[2] = lt.cd[3 * o + 2];
    }
    fl_dst[lane] = (uint8_t)lt.tags;                 // byte j of row r's tag word is byte `lane` of the octet's 32
    fl_dst[32 + lane] = (uint8_t)(lt.tags >> 8);
  } else {
    uint2* c = reinterpret_cast<uint2*>(cd_dst + 24 * lane);
    c[0] = make_uint2(lt.cd[0], lt.cd[1]); c[1] = make_uint2(lt.cd[2], lt.cd[3]); c[2] = make_uint2(lt.cd[4], lt.cd[5]);
    // byte r >> 1 of a row's tag word: the even lane's two groups below the odd one's; the even lane writes tokens 2j, 2j + 1, the odd one the others
    const int j = lane & 3, r = lane >> 2;
    const u32 other = __shfl_xor_sync(FULLM, lt.tags, 4);
    const u32 lo = (r & 1) ? other : lt.tags, hi = (r & 1) ? lt.tags : other;
    const int sh = (r & 1) ? 8 : 0;
    uint8_t* f = fl_dst + 4 * (2 * j + ((r & 1) ? 8 : 0)) + (r >> 1);
    f[0] = (uint8_t)(((lo >> sh) & 15u) | (((hi >> sh) & 15u) << 4));
    f[4] = (uint8_t)(((lo >> (sh + 4)) & 15u) | (((hi >> (sh + 4)) & 15u) << 4));
  }
}

// Write the tile's escape bytes at esc_dst + (tile-relative position), rows in token order, groups ascending.  The tile is still staged in
// ws.xs: a raw group's payload is made from there, in a loop that most lanes never enter (under 1 % of the groups are raw).
template <int KIND_V>
__device__ __forceinline__ void store_tile_escapes(const WarpScratch& ws, const LaneTile& lt, uint8_t* esc_dst, int lane) {
  constexpr int RUN = KIND_V ? 2 : 4;                // groups of a segment
  const int j = lane & 3, r = lane >> 2;
#pragma unroll
  for (int s = 0; s < 8 / RUN; s++) {
    const u32 pw = KIND_V ? lt.pos[s >> 1] : lt.pos[0];
    uint8_t* d = esc_dst + ((s & 1) ? pw >> 16 : pw & 0xFFFFu);
#pragma unroll
    for (int i = 0; i < RUN; i++) {
      const u32 tag = (lt.tags >> (2 * (s * RUN + i))) & 3u;
      if (tag & 1u) *d = (uint8_t)lt.esc1[s * RUN + i];                                      // a raw group's first byte is set right below
      d += tag_esc_bytes(tag);
    }
  }
  for (u32 raw = lt.tags & 0xAAAAu; raw; raw &= raw - 1u) {
    const int bit = __ffs((int)raw) - 1, idx = bit >> 1, s = idx / RUN, g = idx % RUN;
    const u32 below = (lt.tags >> (2 * s * RUN)) & ((1u << (2 * g)) - 1u);
    const u32 pw = KIND_V && (s & 2) ? lt.pos[1] : lt.pos[0];
    uint8_t* d = esc_dst + ((s & 1) ? pw >> 16 : pw & 0xFFFFu) + seg_esc(below);
    u32 sm, e[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (!KIND_V) {
        const u32* p = reinterpret_cast<const u32*>(&ws.xs[(8 * s + r) * XS_STRIDE + 16 * (2 * g + h) + 2 * j]);
        split_bf16x4(p[0], p[4], sm, e[h]);
      } else {
        const uint16_t* p = &ws.xs[v_tok(j, s) * XS_STRIDE + 32 * (2 * g + h) + r];
        split_bf16x4((u32)p[0] | ((u32)p[8] << 16), (u32)p[16] | ((u32)p[24] << 16), sm, e[h]);
      }
    }
    const u64 w = raw_payload(e[0], e[1]);
    d[0] = (uint8_t)w; d[1] = (uint8_t)(w >> 8); d[2] = (uint8_t)(w >> 16); d[3] = (uint8_t)(w >> 24); d[4] = (uint8_t)(w >> 32);
  }
}

// Load the lane's base words for a (kind, base row).
template <int KIND_V>
__device__ __forceinline__ void load_base_words(const uint8_t* b3row, const uint8_t* b4row, int lane, u32* b3w, u32* b4w) {
  if (!KIND_V) { k_base_words(b3row, lane & 3, b3w); k_base_words(b4row, lane & 3, b4w); }
  else { v_base_words(b3row, lane >> 2, b3w); v_base_words(b4row, lane >> 2, b4w); }
}
// Fill the tables of a decoding CTA (any number of threads); the caller synchronises.
template <int KIND_V>
__device__ __forceinline__ u32 fill_decode_tables(DecodeTables& t, const uint8_t* b3row, const uint8_t* b4row) {
  if (threadIdx.x < 32) fill_bases<KIND_V != 0>(t.bases, b3row, b4row, threadIdx.x);
  return (u32)__cvta_generic_to_shared(t.bases);
}
template <bool TRANS> __device__ __forceinline__ void store_matrices(u32 at, int s, u32 w0, u32 w1, u32 w2, u32 w3) {       // the opposite of load_matrices
  if (!TRANS) asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(at + 32 * s), "r"(w0), "r"(w1), "r"(w2), "r"(w3) : "memory");
  else asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(at + 32 * s), "r"(w0), "r"(w1), "r"(w2), "r"(w3) : "memory");
}
// 32 bytes in one load (the address is a multiple of 32)
__device__ __forceinline__ void load_32(u32* w, const void* p) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(p));
}

// A compressed tile on its way: one lane's words as they lie in memory.
template <int KIND_V> struct TileWords {
  static constexpr int SEGS = KIND_V ? 4 : 2;
  u32 sm[16], cd[6], fl[SEGS];
  u32 esc; int n_esc; const uint8_t* esc_src;         // word `lane` of the escape bytes, from the 4-byte boundary at or below the first; how many bytes were asked for
};
// Ask for a tile.  sm / cd / fl: tile-relative sources in global memory; esc_src: the tile's first escape byte.  n_esc: bytes from there on that may be read and are
// likely to be the tile's (0: not known), so that they travel with the rest instead of behind the tags.
template <int KIND_V>
__device__ __forceinline__ void load_tile_words(TileWords<KIND_V>& tw, const uint8_t* sm_src, const uint8_t* cd_src, const uint8_t* fl_src, const uint8_t* esc_src, int n_esc, int lane) {
  const int j = lane & 3;
  constexpr int STEP = KIND_V ? 32 : 1024, SEGS = TileWords<KIND_V>::SEGS;
  u32 (&sm)[16] = tw.sm; u32 (&cd)[6] = tw.cd; u32 (&fl)[SEGS] = tw.fl;
  const uint8_t* s0 = sm_src + (KIND_V ? 64 : 32) * lane;
  {
    const int ofs = (int)(reinterpret_cast<uintptr_t>(esc_src) & 3);
    tw.esc_src = esc_src; tw.n_esc = max(min(n_esc, 128 - ofs), 0); tw.esc = 0u;
    if (tw.n_esc > 0 && 4 * lane < tw.n_esc + ofs) tw.esc = reinterpret_cast<const u32*>(esc_src - ofs)[lane];
  }
  if (!KIND_V) { fl[0] = fl_src[lane]; fl[1] = fl_src[32 + lane]; }                            // byte j of row r's tag word is byte `lane` of the octet's 32
  else {
    const u32* f = reinterpret_cast<const u32*>(fl_src);
#pragma unroll
    for (int t = 0; t < SEGS; t++) fl[t] = f[v_tok(j, t)];
  }
  if ((reinterpret_cast<uintptr_t>(sm_src) & 31) == 0) { load_32(sm, s0); load_32(sm + 8, s0 + STEP); }
  else {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint4 a = *reinterpret_cast<const uint4*>(s0 + h * STEP), b = *reinterpret_cast<const uint4*>(s0 + h * STEP + 16);
      sm[8 * h] = a.x; sm[8 * h + 1] = a.y; sm[8 * h + 2] = a.z; sm[8 * h + 3] = a.w; sm[8 * h + 4] = b.x; sm[8 * h + 5] = b.y; sm[8 * h + 6] = b.z; sm[8 * h + 7] = b.w;
    }
  }
  if (!KIND_V) {
#pragma unroll
    for (int i = 0; i < 6; i++) cd[i] = reinterpret_cast<const u32*>(cd_src + (i / 3) * 384 + 12 * lane)[i % 3];
  } else {
#pragma unroll
    for (int i = 0; i < 3; i++) { const uint2 c = reinterpret_cast<const uint2*>(cd_src + 24 * lane)[i]; cd[2 * i] = c.x; cd[2 * i + 1] = c.y; }
  }
}
// Rebuild the tile into ws.xs (natural channel order, bf16 bits).  The escape bytes that did not come with the rest are fetched with one coalesced load as soon as the
// tags say how many there are (a load per group waited for the one before it at every raw group's branch).  The fragments go to shared memory by
// stmatrix.  most: escape bytes that the scratch behind ws has room for; less than TILE_MAX_ESC only where no tile has more (tags that say otherwise make wrong values and nothing else).
// All of a tile's escape bytes are staged, so that a group reads its own without asking whether it has one, and whether any lane's group is raw is asked once per tile: 771 -> 699 (K) and 788 -> 776
// warp instructions per tile, most of them in branches and 64-bit addresses.  [8, 65536, 128] K and V 88.2 -> 85.7 us;  blocks of 32768 tokens 44.7 -> 43.3, of 512 3.5 -> 3.2.  A second copy of the
// groups for escape bytes in global memory beside them spilled (93), and so did more than one tile per warp of the block decoder.  Tiles of many escape bytes have asynchronous copies of
// them in flight together: by a load and a store per 128 bytes, one behind the other, values of random bits (1280 bytes a tile) took 80.6 us, [8, 32768, 128] K and V, read where they lie 59.4, now 59.2.
// Without the rebuild, loads and stores alone, the pages of 65536 tokens take 80.
template <int KIND_V>
__device__ __forceinline__ void decode_tile_warp(WarpScratch& ws, TileWords<KIND_V>& tw, u32 bases, int lane, int most = TILE_MAX_ESC) {
  const int j = lane & 3, r = lane >> 2;
  constexpr int SEGS = TileWords<KIND_V>::SEGS;
  u32 tags, total, none, pos[SEGS];
  u32 (&sm)[16] = tw.sm; u32 (&cd)[6] = tw.cd; u32 (&fl)[SEGS] = tw.fl;
  const uint8_t* esc_src = tw.esc_src;
  if (!KIND_V) {
    u32 kp, nv[2];
    tile_positions<true, false>(fl[0], fl[1], 0u, 0u, 0u, 0u, j, kp, total, nv, none);
    tags = fl[0] | (fl[1] << 8); pos[0] = kp & 0xFFFFu; pos[1] = kp >> 16;
  } else {
#pragma unroll
    for (int t = 0; t < SEGS; t++) fl[t] = (fl[t] >> (4 * r)) & 15u;
    u32 vp[2];
    tile_positions<false, true>(0u, 0u, fl[0], fl[1], fl[SEGS - 2], fl[SEGS - 1], j, none, none, vp, total);
    tags = fl[0] | (fl[1] << 4) | (fl[SEGS - 2] << 8) | (fl[SEGS - 1] << 12);
#pragma unroll
    for (int t = 0; t < SEGS; t++) pos[t] = t & 1 ? vp[t >> 1] >> 16 : vp[t >> 1] & 0xFFFFu;
  }
  const int n = (int)((total & 0xFFFFu) + (total >> 16)), ofs = (int)(reinterpret_cast<uintptr_t>(esc_src) & 3);
  __syncwarp();                                      // the scratch is no longer in use
  {
    const u32* g = reinterpret_cast<const u32*>(esc_src - ofs);
    u32* const to = reinterpret_cast<u32*>(&ws + 1);
    const int have = tw.n_esc > 0 ? (tw.n_esc + ofs + 3) >> 2 : 0;       // words that came with the rest
    if (lane < have) to[lane] = tw.esc;
    const int end = n > 0 ? min(n, most) + ofs : 0;
    int i = have + lane;
    if (4 * i < end) to[i] = g[i];
    if (4 * (have + 32) < end) {                     // (the same in all lanes) many escape bytes: all of them on their way at once
      const u32 at = (u32)__cvta_generic_to_shared(to);
      for (i += 32; 4 * i < end; i += 32) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(at + 4u * (u32)i), "l"(g + i) : "memory");
      async_commit();
      async_wait<0>();
    }
  }
  const u32 esc0 = (u32)__cvta_generic_to_shared(&ws + 1) + (u32)ofs;
#pragma unroll
  for (int i = 0; i < SEGS; i++) pos[i] = esc0 + min(pos[i], (u32)most);
  const u32 raws = __reduce_or_sync(FULLM, tags & 0xAAAAu);
  __syncwarp();
  const u32 at = matrix_row_address(ws, lane);
#pragma unroll
  for (int g = 0; g < (KIND_V ? 2 : 4); g++) {
    u32 f[SEGS][4];
    const u32x4 bw = lds_u128(bases + (KIND_V ? BASES_V + 32 * r : 64 * j) + 16 * g);
#pragma unroll
    for (int i = 0; i < SEGS; i++) {
      constexpr int PER = 8 / SEGS;                  // groups of a segment
      const int b = 3 * (PER * i + g);               // byte of the group's codes in the lane's 24
      const u32 z = b == 0 ? group_codes<0>(cd) : b == 3 ? group_codes<3>(cd) : b == 6 ? group_codes<6>(cd) : b == 9 ? group_codes<9>(cd) :
                    b == 12 ? group_codes<12>(cd) : b == 15 ? group_codes<15>(cd) : b == 18 ? group_codes<18>(cd) : group_codes<21>(cd);
      decode_group_dev(sm[2 * (PER * i + g)], sm[2 * (PER * i + g) + 1], z, tags >> (2 * (PER * i + g)), pos[i], (raws >> (2 * (PER * i + g)) & 2u) != 0u, bw, f[i]);
    }
    if (!KIND_V) {
#pragma unroll
      for (int h = 0; h < 2; h++) store_matrices<false>(at, 2 * g + h, f[0][2 * h], f[0][2 * h + 1], f[1][2 * h], f[1][2 * h + 1]);
    } else {                                         // word q of a token: channels 8(8g + 2q) + r and 8(8g + 2q + 1) + r; a transposed matrix wants one channel of tokens 2j and 2j + 1
#pragma unroll
      for (int q = 0; q < 4; q++)
        store_matrices<true>(at, 4 * g + q, prmt(f[0][q], f[1][q], 0x5410), prmt(f[0][q], f[1][q], 0x7632), prmt(f[SEGS - 2][q], f[SEGS - 1][q], 0x5410), prmt(f[SEGS - 2][q], f[SEGS - 1][q], 0x7632));
    }
  }
  __syncwarp();
}

// Copy the first nvalid rows of ws.xs to a [*, 128] bf16 matrix (16-byte stores).
__device__ __forceinline__ void unstage_rows(const WarpScratch& ws, uint16_t* dst, long row_stride, int nvalid, int lane) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    int c = lane + 32 * k, row = c >> 4, col = (c & 15) * 8;
    if (row < nvalid) *reinterpret_cast<uint4*>(dst + (long)row * row_stride + col) = *reinterpret_cast<const uint4*>(&ws.xs[row * XS_STRIDE + col]);
  }
}

}  // namespace gaac
