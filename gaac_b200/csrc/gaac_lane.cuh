// Device pieces that the encoder and the decoder share: where a lane's escape bytes lie, and where the rebuild of a group gets its addends from; loads and
// stores of shared memory.  The arithmetic itself is in gaac_tile.h.
#pragma once
#include <cuda_runtime.h>
#include "gaac_tile.h"

namespace gaac {

constexpr unsigned FULLM = 0xffffffffu;

// one step of an inclusive scan over a warp: v += v of the lane `d` below, where there is one
__device__ __forceinline__ void scan_step(u32& v, int d) {
  asm volatile("{\n .reg .pred p;\n .reg .u32 t;\n shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n @p add.u32 %0, %0, t;\n}\n" : "+r"(v) : "r"(d));
}
// ---- escape positions of a lane's segments inside the tile side.
// K: the lanes of an octet are in the order of the tile's escape bytes, so ONE warp scan over both octets' segment sizes (packed in a word) gives
//    every lane its two positions (kpos, low and high half).  k0, k1: tags of the lane's four groups in each octet (8 bits).
// V: a scan over the lanes of equal j (one byte per token: a row has at most 80 escape bytes) places a lane inside its four rows, then a scan
//    over j (two 16-bit sums: tokens 0..7 and 8..15) places the rows inside the tile.  v0..v3: tags of the lane's two groups (4 bits) in
//    tokens 2j, 2j + 1, 2j + 8, 2j + 9; vpos[0]: positions of the first two of them (low and high half), vpos[1]: of the last two.
// ktotal, vtotal: escape bytes of the first eight and the last eight tokens, in the low and the high half.
template <bool HAS_K, bool HAS_V>
__device__ __forceinline__ void tile_positions(u32 k0, u32 k1, u32 v0, u32 v1, u32 v2, u32 v3, int j, u32& kpos, u32& ktotal, u32 (&vpos)[2], u32& vtotal) {
  u32 kown = 0u, vown = 0u;
  if (HAS_K) kown = mad_k<65536u>(seg_esc(k1), seg_esc(k0));
  if (HAS_V) vown = mad_k<16777216u>(seg_esc(v3), mad_k<65536u>(seg_esc(v2), mad_k<256u>(seg_esc(v1), seg_esc(v0))));
  u32 kinc = kown, vinc = vown;
  if (HAS_K) { scan_step(kinc, 1); scan_step(kinc, 2); }
#pragma unroll
  for (int d = 4; d < 32; d <<= 1) { if (HAS_K) scan_step(kinc, d); if (HAS_V) scan_step(vinc, d); }
  if (HAS_K) {
    ktotal = __shfl_sync(FULLM, kinc, 31);
    kpos = kinc - kown + (ktotal << 16);                                                     // the second octet's escape bytes follow the first's
  }
  if (HAS_V) {
    const u32 rows = __shfl_sync(FULLM, vinc, 28 + j), before = vinc - vown;                 // row totals; this lane's share starts `before` into its rows
    const u32 sum = (rows & 0x00FF00FFu) + ((rows >> 8) & 0x00FF00FFu);                     // tokens 2j, 2j + 1 | tokens 2j + 8, 2j + 9
    u32 js = sum;
    { const u32 v = __shfl_up_sync(FULLM, js, 1, 4); if (j >= 1) js += v; }
    { const u32 v = __shfl_up_sync(FULLM, js, 2, 4); if (j >= 2) js += v; }
    vtotal = __shfl_sync(FULLM, js, 3, 4);
    const u32 jb = js - sum + (vtotal << 16);                                                // where rows 2j and 2j + 8 start
    vpos[0] = prmt(jb, 0u, 0x1010) + prmt(before, 0u, 0x4140) + ((rows & 0xFFu) << 16);
    vpos[1] = prmt(jb, 0u, 0x3232) + prmt(before, 0u, 0x4342) + (rows & 0x00FF0000u);
  }
}

// ---- group decoder
constexpr int BASES_V = 256, BASES_BYTES = 512;      // base words of K, of V behind them

__device__ __forceinline__ u32 lds_u8(u32 a) { u32 v; asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ u32 lds_u32(u32 a) { u32 v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ u32x2 lds_u64(u32 a) { u32x2 v; asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ u32x4 lds_u128(u32 a) { u32x4 v; asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
__device__ __forceinline__ void sts_u16(u32 a, u32 v) { asm volatile("{\n .reg .u16 t;\n cvt.u16.u32 t, %1;\n st.shared.u16 [%0], t;\n}" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_u64(u32 a, u32 x, u32 y) { asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory"); }
__device__ __forceinline__ void sts_u128(u32 a, u32 x, u32 y, u32 z, u32 w) { asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory"); }
// Rebuild one group (two sign/mantissa words) into four bf16x2 words; z as group_codes leaves it, tg = tag in the low bits, esc = where its escape bytes are (a shared-memory address,
// which may be read in any case), advanced past them.  raws: some lane's group is raw (the same in all lanes).
__device__ __forceinline__ void decode_group_dev(u32 sm_lo, u32 sm_hi, u32 z, u32 tg, u32& esc, bool raws, const u32x4& bw, u32 out[4]) {
  const u32 m1 = tg & 1u, eb = lds_u8(esc) * m1;      // promoted (tags are 0, 1 or 3)
  u32x2 x = byte_addends(eb);
  if (raws) {
    if (tg & 2u) {
      x = raw_addends(lds_u32(esc & ~3u), lds_u32((esc & ~3u) + 4u), 8u * (esc & 3u), mad(m1, bw.z, bw.x), mad(m1, bw.w, bw.y));
      esc += 4u;
    }
  }
  esc += m1;
  rebuild_group(sm_lo, sm_hi, z, m1, bw, x, out);
}

// ---- base words of a side, {b3lo, b3hi, b4lo - b3lo, b4hi - b3hi} per group (16 bytes; K: lane class jj, group gg at 64 * jj + 16 * gg; V: lane class rr,
// group gg at 32 * rr + 16 * gg).  Thread t < 32 makes word t of the 32 half groups: eight byte loads that do not wait for one another.
template <bool VSIDE>
__device__ __forceinline__ void fill_bases(uint8_t* bases, const uint8_t* b3, const uint8_t* b4, int t) {
  const u32 w3 = half_group_word<VSIDE>(b3, t), w4 = half_group_word<VSIDE>(b4, t);
  u32* o = reinterpret_cast<u32*>(bases + (VSIDE ? BASES_V : 0) + 16 * (t >> 1)) + (t & 1);
  o[0] = w3; o[2] = w4 - w3;
}

}  // namespace gaac
