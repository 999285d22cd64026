// Lane-level view of a GAAC tile (16 tokens x 128 channels): what one lane of a warp encodes or rebuilds.
// Everything here is lane-local and __host__ __device__, and it is what the kernels run: the test-suite drives the same functions on the CPU,
// with plain loops in the place of the warp's scans, its matrix loads and stores and its shared memory.
//
// Storage order (reference: gaac/codec.py:29-67):
//   K tile = two octets of 8 tokens.  Lane l of octet o owns token 8o + (l >> 2) and, with j = l & 3, stored positions
//     [32j, 32j+32): position 32j + 4s + q  <->  channel 16s + 2j + {0,1,8,9}[q].  Its 32 sign/mantissa bytes sit at
//     o*1024 + 32l, its 12 code bytes at o*384 + 12l.  Groups of the lane: 4j + g, g = 0..3 (positions 8g..8g+7 of the lane).
//   V tile: lane l, j = l & 3, r = l >> 2 owns tokens (2j, 2j+1, 2j+8, 2j+9) and stored positions [16r, 16r+16):
//     position 16r + n  <->  channel 8n + r.  Token slot t: 16 sign/mantissa bytes at 64l + 16t, 6 code bytes at 24l + 6t.
//     Groups of the lane: 2r + g, g = 0..1.
#pragma once
#include "gaac_swar.h"

namespace gaac {

// ---- per-lane base words ---------------------------------------------------------------------------------------
// K lane j: word s = bases of channels 16s + 2j + {0,1,8,9}                                      gaac/kernel.py:70-72
GAAC_HD void k_base_words(const uint8_t* row, int j, u32 w[8]) {
  for (int s = 0; s < 8; s++) {
    int d0 = 16 * s + 2 * j;
    w[s] = (u32)row[d0] | ((u32)row[d0 + 1] << 8) | ((u32)row[d0 + 8] << 16) | ((u32)row[d0 + 9] << 24);
  }
}
// V lane class r: word w = bases of channels 8(4w + i) + r, i = 0..3                              gaac/kernel.py:73-75
GAAC_HD void v_base_words(const uint8_t* row, int r, u32 w[4]) {
  for (int i = 0; i < 4; i++)
    w[i] = (u32)row[32 * i + r] | ((u32)row[32 * i + 8 + r] << 8) | ((u32)row[32 * i + 16 + r] << 16) | ((u32)row[32 * i + 24 + r] << 24);
}

// Word t (0..31) of a side's 32 half groups, in the order in which they are read: K: 8 * (lane & 3) + s, V: 4 * (lane >> 2) + w.  Four byte loads that do not
// wait for one another.
template <bool VSIDE> GAAC_HD u32 half_group_word(const uint8_t* row, int t) {
  const int d0 = VSIDE ? 32 * (t & 3) + (t >> 2) : 16 * (t & 7) + 2 * (t >> 3), d1 = d0 + (VSIDE ? 8 : 1), d2 = d0 + (VSIDE ? 16 : 8), d3 = d0 + (VSIDE ? 24 : 9);
  return (u32)row[d0] | (u32)row[d1] << 8 | (u32)row[d2] << 16 | (u32)row[d3] << 24;
}

// ---- encode ----------------------------------------------------------------------------------------------------
// Four groups of 24 code bits (bits 24..31 ignored) -> 96 bits
GAAC_HD void join_codes(u32 c0, u32 c1, u32 c2, u32 c3, u32* cd) {
  cd[0] = prmt(c0, c1, 0x4210); cd[1] = prmt(c1, c2, 0x5421); cd[2] = prmt(c2, c3, 0x6542);
}
GAAC_HD int tag_esc_bytes(u32 tag) { return (int)(tag & 1u) + 2 * (int)(tag & 2u); }   // 0, 1, 5 for tags 0, 1, 3

// ---- decode ----------------------------------------------------------------------------------------------------
struct u32x4 { u32 x, y, z, w; };
struct u32x2 { u32 x, y; };
// What escape byte b adds to the exponents of its group: of elements 0..3, 4..7
GAAC_HD u32x2 byte_addends(u32 b) { return u32x2{spread_bit4(b & 15u), spread_bit4(b >> 4)}; }
// The 24 code bits of a group, picked out of two neighbouring words by one byte permute that already puts codes 4..7 at the top:
// bits 0..11 = codes 0..3, bits 20..31 = codes 4..7 (B = byte offset of the group in the lane's code string).
template <int B> GAAC_HD u32 group_codes(const u32* cd) {
  constexpr int i = B & 3;
  constexpr u32 sel = (u32)i | (u32)(i + 1) << 4 | (u32)(i + 1) << 8 | (u32)(i + 2) << 12;
  return prmt(cd[B >> 2], i >= 2 ? cd[(B >> 2) + 1] : 0u, sel);
}
// What a raw group adds to its codes: its payload's five bytes lie in (w1:w0) from bit sh (0, 8, 16, 24), five bits per element.  blo, bhi: the base words
// that rebuild_group adds to every promoted group, taken off here (e = code | hi5 << 3, the base must not contribute).
GAAC_HD u32x2 raw_addends(u32 w0, u32 w1, u32 sh, u32 blo, u32 bhi) {
  const u32 lo = funnel_r(w0, w1, (int)sh), hi = w1 >> sh;               // bytes 0-3 and byte 4 of the payload
  return u32x2{spread_hi5(lo & 0xFFFFFu) - blo, spread_hi5(funnel_r(lo, hi, 20) & 0xFFFFFu) - bhi};
}
// Rebuild one group (two sign/mantissa words) into four bf16x2 words: z as group_codes leaves it; m1 = 1 for a promoted group; bw = {3-bit-window base words of
// the two half groups, what the 4-bit-window ones are above them}; x = the group's addends, of byte_addends or raw_addends.
GAAC_HD void rebuild_group(u32 sm_lo, u32 sm_hi, u32 z, u32 m1, const u32x4& bw, const u32x2& x, u32 out[4]) {
  const u32 blo = mad(m1, bw.z, bw.x), bhi = mad(m1, bw.w, bw.y);
  // four 3-bit codes -> four bytes in two steps; each step moves the upper fields with a multiply-add: (t & M) * (2^k - 1) + t
  const u32 th = z >> 20;
  const u32 xl = mad_k<1023u>(z & 0xFC0u, z & 0xFFFu), xh = mad_k<1023u>(th & 0xFC0u, th);
  bf16x4(sm_lo, mad_k<31u>(xl & 0x00380038u, xl) + blo + x.x, out[0], out[1]);
  bf16x4(sm_hi, mad_k<31u>(xh & 0x00380038u, xh) + bhi + x.y, out[2], out[3]);
}

// ---- decode, the form of the attention kernels.  A rebuilt word there may hold any two elements of a group, as long as the other operand of the matrix product
// has the same two, so the codes go into bytes in two steps for the whole group ({0, 1}, {2, 3}, {4, 5}, {6, 7}: code_bytes), the exponents are made in two
// words, of the even and of the odd elements, and a word pairs elements that lie four apart: bytes 0 and 2 of a word of exponents land on the exponent fields
// of a bf16 pair when it is shifted up by 7, bytes 1 and 3 when it is shifted down by 1, whatever else the shift brings along is covered by the sign and
// mantissa bits, and those come from one byte permute.  
// The codes of a group, two to a byte, at bits 0..5; the bits above are anything (B = byte offset of the group in the lane's code string).  A step is a shift and a select: with the fields
// masked and moved by multiply-adds a group took one operation of the ALU more (12 of 1010 instructions per tile pair; 65536 tokens 49.8 -> 49.3 us, paged 16 x 4096..65536 406 -> 404).
template <int B> GAAC_HD u32 code_bytes(const u32* cd) {
  constexpr int i = B & 3;
  u32 t;                                                                 // codes 0..3 at bits 0..11, 4..7 at bits 16..27
  if (i == 1) t = bits_of(cd[B >> 2] >> 8, cd[B >> 2] >> 4, 0xFFFu);
  else {
    const u32 z = i ? prmt(cd[B >> 2], cd[(B >> 2) + (i ? 1 : 0)], i == 2 ? 0x5432 : 0x6543) : cd[B >> 2];      // the upper byte is the next group's
    t = bits_of(z, mad_k<16u>(z, 0u), 0xFFFu);
  }
  return bits_of(t, mad_k<4u>(t, 0u), 0x003F003Fu);
}
// Words of the bases {3-bit window: even elements, odd elements; what the 4-bit window is above them: even, odd} of group t of a side's 16 (K: 4 * (lane & 3)
// + group, V: 2 * (lane >> 2) + group)
template <bool VSIDE> GAAC_HD u32x4 pair_base_words(const uint8_t* row3, const uint8_t* row4, int t) {
  const u32 a3 = half_group_word<VSIDE>(row3, 2 * t), b3 = half_group_word<VSIDE>(row3, 2 * t + 1), a4 = half_group_word<VSIDE>(row4, 2 * t), b4 = half_group_word<VSIDE>(row4, 2 * t + 1);
  const u32 e3 = prmt(a3, b3, 0x6420), o3 = prmt(a3, b3, 0x7531);
  return u32x4{e3, o3, prmt(a4, b4, 0x6420) - e3, prmt(a4, b4, 0x7531) - o3};
}
// What an escape byte adds to the exponents of its group: 8 in byte k for bit 2k (even elements) and for bit 2k + 1 (odd ones)
GAAC_HD u32x2 pair_addends(u32 b) {
  const u32 lo = spread_bit4(b & 15u), hi = spread_bit4(b >> 4);
  return u32x2{prmt(lo, hi, 0x6420), prmt(lo, hi, 0x7531)};
}
// The upper five bits of the exponents of a raw group's even and odd elements, from its payload of 8 x 5 bits: bits 0..31, and from bit 32 on (more bits may follow).  Two fields
// side by side at bits 0 and 16 of a word, for the first four and for the last, and one byte permute each for the even and the odd ones.
GAAC_HD u32x2 pair_payload(u32 lo, u32 byte4) {
  const u32 z = funnel_r(lo, byte4, 20), a = bits_of(lo, mad_k<64u>(lo, 0u), 0x3FFu), b = bits_of(z, mad_k<64u>(z, 0u), 0x3FFu);
  return u32x2{mad_k<8u>(prmt(a, b, 0x6420), 0u) & 0xF8F8F8F8u, prmt(a >> 2, b >> 2, 0x6420) & 0xF8F8F8F8u};
}
// The same for a raw group, whose payload (8 x 5 bits) lies in (w1:w0) from bit sh (0, 8, 16, 24): the upper five bits of the exponents.  No base must contribute:
// the caller takes off what rebuild_pairs adds.
GAAC_HD u32x2 pair_raw_addends(u32 w0, u32 w1, u32 sh) {
  return pair_payload(funnel_r(w0, w1, (int)sh), w1 >> sh);
}
// out[i] = elements i and i + 4.  u: code_bytes; m: what the bases' second half counts (1 for a promoted group); x: the addends.
GAAC_HD void rebuild_pairs(u32 sm_lo, u32 sm_hi, u32 u, u32 m, const u32x4& bw, const u32x2& x, u32 out[4]) {
  const u32 ev = (u & 0x07070707u) + mad(m, bw.z, bw.x) + x.x, od = mad_shr<3>(u & 0x38383838u, mad(m, bw.w, bw.y)) + x.y;
  out[0] = bits_of(prmt(sm_lo, sm_hi, 0x4400), mad_k<128u>(ev, 0u), 0x807F807Fu);
  out[1] = bits_of(prmt(sm_lo, sm_hi, 0x5511), mad_k<128u>(od, 0u), 0x807F807Fu);
  out[2] = bits_of(prmt(sm_lo, sm_hi, 0x6622), ev >> 1, 0x807F807Fu);
  out[3] = bits_of(prmt(sm_lo, sm_hi, 0x7733), od >> 1, 0x807F807Fu);
}
// ---- escape bytes of four neighbouring groups of a row (a segment), by its tag byte t.  Segment words hold a 16-bit index per group: NO_ESC for a group without
// escape byte, 256 + byte for a promoted one; entry `index` of the addend table is what to add, index >> 8 the m of rebuild_pairs.  {x: selector of 16 bits that picks the
// indexes of groups 0, 1 out of the segment's first four escape bytes and SEG_CONST, above it the segment's escape bytes; y: the selector of groups 2, 3}, since a permute takes the
// lower half of a selector.  The selectors are right for the groups up to the segment's first raw one; raw_items are the others.
constexpr u32 NO_ESC = 255u, SEG_CONST = 0x000100FFu;
GAAC_HD u32x2 segment_entry(u32 t) {
  u32 sel = 0u, at = 0u;
  for (int g = 0; g < 4; g++) {
    const u32 tag = (t >> (2 * g)) & 3u;
    sel |= (tag & 1u ? 0x60u | at : 0x54u) << (8 * g);
    at += tag & 1u;
  }
  return u32x2{(sel & 0xFFFFu) | seg_esc(t) << 16, sel >> 16};
}
// Groups of a row with tag word fl that the selectors leave out: the raw ones and the promoted ones behind a raw one of their segment, at their lower tag bits.
GAAC_HD u32 raw_items(u32 fl) {
  const u32 r = (fl >> 1) & fl & 0x55555555u;
  return (r | (0x80808080u - r)) & fl & 0x55555555u;                     // bits 0..6 of a byte's 0x80 - r: those of -r, ones above the lowest one of r
}

}  // namespace gaac
