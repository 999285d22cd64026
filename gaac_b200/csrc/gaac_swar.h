// Byte-SWAR building blocks of the GAAC tile format, shared by every kernel (encoder, decoder, fused attention).
// All functions are __host__ __device__: the test-suite runs them on the CPU.
//
// Format facts used here (reference: gaac/codec.py:1-18,139-172; gaac/kernel.py:29-46):
//   bf16 bits x  ->  e = (x >> 7) & 0xFF,  sm = ((x >> 8) & 0x80) | (x & 0x7F)
//   group of 8 stored positions: tier 0 -> e = base3 + code, tier 1 -> e = base4 + code + 8*bit4, tier 2 -> e = code | hi5 << 3
//   tags: 2 bits per group in a u32 per row (bit0 = promoted, bit1 = raw); escape bytes: tier 1 -> 1, tier 2 -> 5.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define GAAC_HD __host__ __device__ __forceinline__
#else
#define GAAC_HD inline
#endif

namespace gaac {

typedef uint32_t u32;
typedef uint64_t u64;

constexpr int D = 128;          // head dim
constexpr int T = 16;           // tokens per tile
constexpr int CB = 48;          // code bytes per row
constexpr int TILE_SM = T * D;  // 2048
constexpr int TILE_CD = T * CB; // 768
constexpr int TILE_MAX_ESC = 1280;
constexpr int SLOT_CD_OFF = 2048, SLOT_FL_OFF = 2816, SLOT_OVF_OFF = 2880;   // paged tile slot layout (gaac/vllm/store.py:18)
// Mode-table entry m < 0 of the paged layout: the rows are in raw tile raw_tile(m) of the pool, ~m when the block owns that tile.  A block that found the
// pool empty owns none: its entry is ~RAW_NONE, its rows are lost, readers get those of tile 0.
constexpr int RAW_NONE = 1 << 30;

// ---- portable intrinsics ---------------------------------------------------------------------------------------
GAAC_HD u32 prmt(u32 a, u32 b, u32 sel) {
#if defined(__CUDA_ARCH__)
  return __byte_perm(a, b, sel);
#else
  u64 pool = (u64)a | ((u64)b << 32);
  u32 r = 0;
  for (int i = 0; i < 4; i++) r |= (u32)((pool >> (8 * ((sel >> (4 * i)) & 7))) & 0xFF) << (8 * i);
  return r;
#endif
}
GAAC_HD u32 funnel_r(u32 lo, u32 hi, int sh) {          // (hi:lo) >> sh, 0 <= sh < 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, sh);
#else
  return sh ? (u32)((((u64)hi << 32) | lo) >> sh) : lo;
#endif
}
GAAC_HD int raw_tile(int m) { return ~m & (RAW_NONE - 1); }
// the bits of a where the mask has ones, those of b elsewhere (one instruction; the compiler needs two for the and/and/or form)
GAAC_HD u32 bits_of(u32 a, u32 b, u32 mask) {
#if defined(__CUDA_ARCH__)
  u32 d; asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(d) : "r"(a), "r"(b), "r"(mask)); return d;
#else
  return (a & mask) | (b & ~mask);
#endif
}
GAAC_HD int popc(u32 x) {
#if defined(__CUDA_ARCH__)
  return __popc(x);
#else
  return __builtin_popcount(x);
#endif
}

// ---- multiply-adds.  Logic ops (LOP3 / PRMT / SHF) run on the ALU pipe, whose rate is half the issue rate, so shifts that can be merged with an add are
// written as multiply-adds (FMA pipe)
template <u32 K> GAAC_HD u32 mad_k(u32 a, u32 c) {
#if defined(__CUDA_ARCH__)
  u32 d; asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "n"(K), "r"(c)); return d;
#else
  return a * K + c;
#endif
}
GAAC_HD u32 mad(u32 a, u32 b, u32 c) {
#if defined(__CUDA_ARCH__)
  u32 d; asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d;
#else
  return a * b + c;
#endif
}
// (a >> S) + c
template <int S> GAAC_HD u32 mad_shr(u32 a, u32 c) {
#if defined(__CUDA_ARCH__)
  u32 d; asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "n"(1u << (32 - S)), "r"(c)); return d;
#else
  return (a >> S) + c;
#endif
}

// byte B of a, times K (K < 256), plus c: one dot product of four bytes, where a byte's extraction is an instruction of the ALU and the multiply-add another
template <int B, u32 K> GAAC_HD u32 mad_byte(u32 a, u32 c) {
#if defined(__CUDA_ARCH__)
  u32 d; asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(K << (8 * B)), "r"(c)); return d;
#else
  return ((a >> (8 * B)) & 0xFFu) * K + c;
#endif
}
// the same for half H (0: the lower, 1: the upper) of a
template <int H, u32 K> GAAC_HD u32 mad_half(u32 a, u32 c) {
#if defined(__CUDA_ARCH__)
  u32 d; asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(K << (8 * H)), "r"(c)); return d;
#else
  return ((a >> (16 * H)) & 0xFFFFu) * K + c;
#endif
}

// ---- tags -> escape byte counts --------------------------------------------------------------------------------
// escape bytes of a row with tag word fl (tier 1 -> 1 byte, tier 2 -> 5 bytes)                  gaac/kernel.py:46
GAAC_HD int row_esc_bytes(u32 fl) { return popc(fl & 0x55555555u) + 4 * popc(fl & 0xAAAAAAAAu); }
// .. of the groups whose tag bits are in `below`
GAAC_HD u32 esc_below(u32 fl, u32 below) { return (u32)popc(fl & below & 0x55555555u) + 4u * (u32)popc(fl & below & 0xAAAAAAAAu); }
// escape bytes of the groups below bit position `bits` of the tag word                            gaac/kernel.py:29
GAAC_HD int esc_prefix(u32 fl, int bits) {
  u32 low = bits >= 32 ? fl : (fl & ((1u << bits) - 1u));
  return popc(low & 0x55555555u) + 4 * popc(low & 0xAAAAAAAAu);
}

// Escape bytes of up to four groups whose tags are t (upper bits clear): one for a promoted group (tag 01), five for a raw one (11), which
// is one bit per tag bit and three more copies of every upper bit.
GAAC_HD u32 seg_esc(u32 t) { return (u32)popc((t & 0xAAu) * 0x01010100u + t); }

// ---- decode side -----------------------------------------------------------------------------------------------
// four 1-bit flags at bits 0..3 of n (n < 16) -> 8 * flag per byte (the 4th bit of a 4-bit window code)
GAAC_HD u32 spread_bit4(u32 n) { return (n * 0x01020408u) & 0x08080808u; }
// four 5-bit fields at bits 0..19 of u (the others clear) -> field << 3 per byte (raw-tier exponent high bits)
GAAC_HD u32 spread_hi5(u32 u) {
  const u32 y = mad_k<64u>(u & 0xFFC00u, u & 0x3FFu);               // fields 0,1 at bits 0-9, fields 2,3 at bits 16-25
  return mad_k<64u>(y & 0x03E003E0u, (y & 0x001F001Fu) << 3);       // odd fields up 3 more bits, everything << 3
}
// sign/mantissa bytes (4) + exponent bytes (4) -> bf16 pairs (elements 0,1) and (2,3)             gaac/kernel.py:34-36
GAAC_HD void bf16x4(u32 sm4, u32 e4, u32& p01, u32& p23) {
  const u32 eh = e4 >> 1;
  const u32 el = mad_k<128u>(e4, 0u);                                // e4 << 7
  const u32 h4 = bits_of(sm4, eh, 0x80808080u), l4 = bits_of(el, sm4, 0x80808080u);
  p01 = prmt(l4, h4, 0x5140); p23 = prmt(l4, h4, 0x7362);
}

// ---- encode side -----------------------------------------------------------------------------------------------
// low bytes (l4) and high bytes (h4) of four bf16 values -> sign/mantissa bytes and exponent bytes
GAAC_HD void split_bytes4(u32 l4, u32 h4, u32& sm4, u32& e4) {
  sm4 = bits_of(h4, l4, 0x80808080u);
  e4 = bits_of(h4 * 2u, l4 >> 7, 0xFEFEFEFEu);
}
// two bf16 pairs (elements 0,1) (2,3) -> sign/mantissa bytes and exponent bytes
GAAC_HD void split_bf16x4(u32 p01, u32 p23, u32& sm4, u32& e4) { split_bytes4(prmt(p01, p23, 0x6420), prmt(p01, p23, 0x7531), sm4, e4); }
// four channels of two tokens, one word per channel (low half: the first token), -> the same for each token: a byte transpose sorts them by token and by
// low / high byte
GAAC_HD void split_token_pairs(u32 x0, u32 x1, u32 x2, u32 x3, u32& sm_a, u32& e_a, u32& sm_b, u32& e_b) {
  const u32 p = prmt(x0, x1, 0x5140), q = prmt(x2, x3, 0x5140), p2 = prmt(x0, x1, 0x7362), q2 = prmt(x2, x3, 0x7362);
  split_bytes4(prmt(p, q, 0x5410), prmt(p, q, 0x7632), sm_a, e_a);
  split_bytes4(prmt(p2, q2, 0x5410), prmt(p2, q2, 0x7632), sm_b, e_b);
}
// bit 3 of each byte of lo (bits 0-3 of the result) and of hi (bits 4-7): the fields are 8 bits apart, so one multiply brings them side by side
GAAC_HD u32 pack_bit4x2(u32 lo, u32 hi) { return (((hi & 0x08080808u) * 16u + (lo & 0x08080808u)) * 0x00204081u) >> 24; }
// (byte >> 3) of each byte -> 20 bits
GAAC_HD u32 pack_hi5(u32 e4) {
  u32 f = (e4 >> 3) & 0x1F1F1F1Fu;
  return (f & 0x1Fu) | ((f >> 3) & 0x3E0u) | ((f >> 6) & 0x7C00u) | ((f >> 9) & 0xF8000u);
}
// the low three bits of every byte of lo (elements 0-3) and hi (4-7) -> 24 bits, element i at bit 3i; higher bits of the bytes are ignored
// (bits 24 and above of the result are anything).  Fields are moved next to one another by multiplications, 7 of the 11 operations on the ALU, which the encoder keeps busiest; by shifts and selects all
// 11 were: [8, 8192, 128] 9.13 (K) / 8.65 (V) -> 9.01 / 8.47 us, x 65536 45.4 / 44.1 -> 45.1 / 44.0.
GAAC_HD u32 pack_codes8(u32 lo, u32 hi) {
  const u32 yl = mad_k<33u>(lo & 0x07070707u, 0u), yh = mad_k<33u>(hi & 0x07070707u, 0u);                  // two codes side by side at bits 5-10 and at 21-26
  const u32 zl = mad_k<1025u>(yl & 0x07E007E0u, 0u), zh = mad_k<1025u>(yh & 0x07E007E0u, 0u);              // four at bits 15-26
  return bits_of(zl >> 15, zh >> 3, 0x00000FFFu);
}

// Encode one group of 8 stored positions given its exponent bytes (elements 0-3 in e_lo, 4-7 in e_hi) and the bases.
// Returns the tier tag (0, 1, 3); codes24 = 8 x 3-bit codes; esc1 = the escape byte of tier 1 (any value for the other tiers).
// A window is tried with ONE 32-bit subtraction per half group: base tables leave room for their window (3-bit base <= 248, 4-bit base <=
// 240), so "every byte of e - b is below the window" as a plain word difference means that no byte borrowed, which is the same as
// "every exponent lies in its window".  Both windows are tried up front and everything is picked with selects: in a warp some lane
// nearly always needs the 4-bit window.
GAAC_HD u32 encode_group_codes(u32 e_lo, u32 e_hi, u32 b3_lo, u32 b3_hi, u32 b4_lo, u32 b4_hi, u32& codes24, u32& esc1) {
  const u32 d3l = e_lo - b3_lo, d3h = e_hi - b3_hi, d4l = e_lo - b4_lo, d4h = e_hi - b4_hi;
  const bool t0 = ((d3l | d3h) & 0xF8F8F8F8u) == 0, t1 = ((d4l | d4h) & 0xF0F0F0F0u) == 0;
  codes24 = pack_codes8(t0 ? d3l : (t1 ? d4l : e_lo), t0 ? d3h : (t1 ? d4h : e_hi));
  esc1 = pack_bit4x2(d4l, d4h);
  return t0 ? 0u : (t1 ? 1u : 3u);
}
// Escape payload of a raw group: the upper five bits of its eight exponents, 40 bits.
GAAC_HD u64 raw_payload(u32 e_lo, u32 e_hi) { return (u64)pack_hi5(e_lo) | ((u64)pack_hi5(e_hi) << 20); }
}  // namespace gaac
