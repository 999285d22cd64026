// Host emulation of one warp encoding / rebuilding a GAAC tile with the SAME lane-level functions the CUDA kernels run
// (gaac_b200/csrc/gaac_tile.h, gaac_swar.h).  What is warp-level there - matrix loads and stores, the scans that place the escape bytes, the
// tables in shared memory - is plain loops here.
// Built by the test-suite with g++ and driven through ctypes; checks the bit logic without a GPU.
#include <cstring>
#include "../../gaac_b200/csrc/gaac_tile.h"
using namespace gaac;

static int v_tok(int j, int t) { return 2 * j + (t & 1) + 8 * (t >> 1); }
static u32 pair(u32 lo, u32 hi) { return lo | hi << 16; }
// position of a lane's escape bytes: those of the rows before and of the groups below `first` in the row
static int esc_at(const uint32_t* fl, int row, int first) {
  int at = 0;
  for (int i = 0; i < row; i++) at += row_esc_bytes(fl[i]);
  for (int g = 0; g < first; g++) at += (int)seg_esc((fl[row] >> (2 * g)) & 3u);
  return at;
}

extern "C" int emu_encode_tile(int kind_v, const uint16_t* x, int nvalid, const uint8_t* b3row, const uint8_t* b4row,
                               uint8_t* sm_out, uint8_t* cd_out, uint32_t* fl_out, uint8_t* esc_out) {
  static const uint16_t zeros[128] = {};
  auto at = [&](int tok) { return tok < nvalid ? x + 128 * tok : zeros; };
  struct Group { u32 tag, esc1; u64 raw; } groups[16][16];
  for (int lane = 0; lane < 32; lane++) {
    const int j = lane & 3, r = lane >> 2;
    u32 b3w[8], b4w[8], sm[16], cd[6], c24[8];
    if (!kind_v) {
      k_base_words(b3row, j, b3w); k_base_words(b4row, j, b4w);
      for (int o = 0; o < 2; o++) {
        u32 e[8];
        const uint16_t* row = at(8 * o + r);
        for (int s = 0; s < 8; s++) { const uint16_t* p = row + 16 * s + 2 * j; split_bf16x4(pair(p[0], p[1]), pair(p[8], p[9]), sm[8 * o + s], e[s]); }
        for (int g = 0; g < 4; g++) {
          Group& G = groups[8 * o + r][4 * j + g];
          G.tag = encode_group_codes(e[2 * g], e[2 * g + 1], b3w[2 * g], b3w[2 * g + 1], b4w[2 * g], b4w[2 * g + 1], c24[4 * o + g], G.esc1);
          G.raw = raw_payload(e[2 * g], e[2 * g + 1]);
          if (8 * o + r >= nvalid) G.tag = c24[4 * o + g] = 0;
        }
      }
    } else {
      v_base_words(b3row, r, b3w); v_base_words(b4row, r, b4w);
      u32 e[4][4];                                   // [token slot][word]
      for (int i = 0; i < 4; i++)
        for (int th = 0; th < 2; th++) {
          const uint16_t *a = at(2 * j + 8 * th), *b = at(2 * j + 1 + 8 * th);
          u32 w[4];
          for (int q = 0; q < 4; q++) w[q] = pair(a[32 * i + 8 * q + r], b[32 * i + 8 * q + r]);
          split_token_pairs(w[0], w[1], w[2], w[3], sm[8 * th + i], e[2 * th][i], sm[8 * th + 4 + i], e[2 * th + 1][i]);
        }
      for (int t = 0; t < 4; t++)
        for (int g = 0; g < 2; g++) {
          Group& G = groups[v_tok(j, t)][2 * r + g];
          G.tag = encode_group_codes(e[t][2 * g], e[t][2 * g + 1], b3w[2 * g], b3w[2 * g + 1], b4w[2 * g], b4w[2 * g + 1], c24[2 * t + g], G.esc1);
          G.raw = raw_payload(e[t][2 * g], e[t][2 * g + 1]);
          if (v_tok(j, t) >= nvalid) G.tag = c24[2 * t + g] = 0;
        }
    }
    join_codes(c24[0], c24[1], c24[2], c24[3], cd);
    join_codes(c24[4], c24[5], c24[6], c24[7], cd + 3);
    if (!kind_v)
      for (int o = 0; o < 2; o++) { memcpy(sm_out + o * 1024 + 32 * lane, sm + 8 * o, 32); memcpy(cd_out + o * 384 + 12 * lane, cd + 3 * o, 12); }
    else { memcpy(sm_out + 64 * lane, sm, 64); memcpy(cd_out + 24 * lane, cd, 24); }
  }
  int total = 0;
  for (int row = 0; row < 16; row++) {
    fl_out[row] = 0;
    for (int g = 0; g < 16; g++) fl_out[row] |= groups[row][g].tag << (2 * g);
    for (int g = 0; g < 16; g++) {
      const Group& G = groups[row][g];
      uint8_t* d = esc_out + esc_at(fl_out, row, g);
      if (G.tag == 1u) d[0] = (uint8_t)G.esc1;
      if (G.tag == 3u) for (int i = 0; i < 5; i++) d[i] = (uint8_t)(G.raw >> (8 * i));
    }
    total += row_esc_bytes(fl_out[row]);
  }
  return total;
}

// Rebuild as the decoders do it (decode_tile_warp, decode_group_dev): a lane goes along its segments' escape bytes, of which it reads one per group whether the group has it or not.
// esc_in must be readable to the end of the word behind its last byte.
extern "C" void emu_decode_tile(int kind_v, const uint8_t* sm_in, const uint8_t* cd_in, const uint32_t* fl_in, const uint8_t* esc_in, const uint8_t* b3row, const uint8_t* b4row, uint16_t* out) {
  const int SEGS = kind_v ? 4 : 2, PER = 8 / SEGS;
  u32 base[32][2];                                   // {3-bit window, what the 4-bit one is above it} per half group
  for (int t = 0; t < 32; t++) {
    base[t][0] = kind_v ? half_group_word<true>(b3row, t) : half_group_word<false>(b3row, t);
    base[t][1] = (kind_v ? half_group_word<true>(b4row, t) : half_group_word<false>(b4row, t)) - base[t][0];
  }
  for (int lane = 0; lane < 32; lane++) {
    const int j = lane & 3, r = lane >> 2;
    u32 sm[16], cd[6];
    if (!kind_v) for (int o = 0; o < 2; o++) { memcpy(sm + 8 * o, sm_in + o * 1024 + 32 * lane, 32); memcpy(cd + 3 * o, cd_in + o * 384 + 12 * lane, 12); }
    else { memcpy(sm, sm_in + 64 * lane, 64); memcpy(cd, cd_in + 24 * lane, 24); }
    const u32 z[8] = {group_codes<0>(cd), group_codes<3>(cd), group_codes<6>(cd), group_codes<9>(cd), group_codes<12>(cd), group_codes<15>(cd), group_codes<18>(cd), group_codes<21>(cd)};
    for (int s = 0; s < SEGS; s++) {
      const int row = kind_v ? v_tok(j, s) : 8 * s + r, first = kind_v ? 2 * r : 4 * j;
      const uint8_t* esc = esc_in + esc_at(fl_in, row, first);
      for (int g = 0; g < PER; g++) {
        const int idx = PER * s + g, hg = kind_v ? 4 * r + 2 * g : 8 * j + 2 * g;
        const u32 tag = (fl_in[row] >> (2 * (first + g))) & 3u, m1 = tag & 1u;
        const u32x4 bw{base[hg][0], base[hg + 1][0], base[hg][1], base[hg + 1][1]};
        u32x2 x = byte_addends(*esc * m1);
        if (tag & 2u) {
          const u32* a = reinterpret_cast<const u32*>(reinterpret_cast<uintptr_t>(esc) & ~(uintptr_t)3);
          x = raw_addends(a[0], a[1], 8u * (u32)(reinterpret_cast<uintptr_t>(esc) & 3), mad(m1, bw.z, bw.x), mad(m1, bw.w, bw.y));
          esc += 4;
        }
        esc += m1;
        u32 f[4];
        rebuild_group(sm[2 * idx], sm[2 * idx + 1], z[idx], m1, bw, x, f);
        for (int q = 0; q < 4; q++) {
          // K: words 2h, 2h + 1 = channels 16s + 2j (+ 1) and + 8 (+ 1) of s = 2g + h; V: word q = channels 8(8g + 2q) + r and 8(8g + 2q + 1) + r
          const int c = kind_v ? 8 * (8 * g + 2 * q) + r : 16 * (2 * g + (q >> 1)) + 2 * j + 8 * (q & 1);
          out[128 * row + c] = (uint16_t)f[q]; out[128 * row + c + (kind_v ? 8 : 1)] = (uint16_t)(f[q] >> 16);
        }
      }
    }
  }
}

// Rebuild as the attention kernels do it (plan_tile, rebuild_pairs): the tile's segments (four groups of a row) are expanded into indexes of the addend table, a raw group's index is
// that of an entry of its own behind the table, and a word pairs elements that lie four apart.  first_patch: index of the first such entry.
extern "C" int emu_decode_tile_pairs(int kind_v, const uint8_t* sm_in, const uint8_t* cd_in, const uint32_t* fl_in, const uint8_t* esc_in,
                                     const uint8_t* b3row, const uint8_t* b4row, int first_patch, uint16_t* out) {
  static u32x2 addends[65536];
  addends[NO_ESC] = u32x2{0u, 0u};
  for (u32 b = 0; b < 256; b++) addends[256 + b] = pair_addends(b);
  u32x4 base[16];
  for (int t = 0; t < 16; t++) base[t] = kind_v ? pair_base_words<true>(b3row, b4row, t) : pair_base_words<false>(b3row, b4row, t);
  u32 words[16][4][2];                               // segment words of row, quarter
  int raws = 0;
  for (int row = 0; row < 16; row++) {               // a lane's row
    const u32 fl = fl_in[row];
    const uint8_t* const at = esc_in + esc_at(fl_in, row, 0);
    const uint8_t* a = at;
    for (int q = 0; q < 4; q++) {
      const u32x2 e = segment_entry((fl >> (8 * q)) & 0xFFu);
      const u32 four = (u32)a[0] | (u32)a[1] << 8 | (u32)a[2] << 16 | (u32)a[3] << 24;
      words[row][q][0] = prmt(four, SEG_CONST, e.x); words[row][q][1] = prmt(four, SEG_CONST, e.y);
      a += e.x >> 16;
    }
    if (a - at != row_esc_bytes(fl)) return -1;
    uint16_t* const indexes = reinterpret_cast<uint16_t*>(words[row]);
    u32 raw = (fl >> 1) & fl & 0x55555555u, behind = raw_items(fl) & ~raw;
    raws += popc(raw);
    u32 index = (u32)(first_patch + raws);           // behind the row's entries: from the last to the first
    while (raw) {
      const u32 bit = 31u - (u32)__builtin_clz(raw), below = ~(0xFFFFFFFFu << bit);
      raw &= below; index--;
      const uint8_t* const pl = at + esc_below(fl, below);
      const u32* const w = reinterpret_cast<const u32*>(reinterpret_cast<uintptr_t>(pl) & ~(uintptr_t)3);
      const u32x2 x = pair_payload(funnel_r(w[0], w[1], (int)(8 * (reinterpret_cast<uintptr_t>(pl) & 3))), pl[4]);
      const u32 m = index >> 8;
      const u32x4& bw = base[bit >> 1];
      addends[index] = u32x2{x.x - bw.x - m * bw.z, x.y - bw.y - m * bw.w};
      indexes[bit >> 1] = (uint16_t)index;
    }
    while (behind) {
      const u32 bit = 31u - (u32)__builtin_clz(behind), below = ~(0xFFFFFFFFu << bit);
      behind &= below;
      indexes[bit >> 1] = (uint16_t)(256u + at[esc_below(fl, below)]);
    }
  }
  const int SEGS = kind_v ? 4 : 2, PER = 8 / SEGS;
  for (int lane = 0; lane < 32; lane++) {
    const int j = lane & 3, r = lane >> 2;
    u32 sm[16], cd[6];
    if (!kind_v) for (int o = 0; o < 2; o++) { memcpy(sm + 8 * o, sm_in + o * 1024 + 32 * lane, 32); memcpy(cd + 3 * o, cd_in + o * 384 + 12 * lane, 12); }
    else { memcpy(sm, sm_in + 64 * lane, 64); memcpy(cd, cd_in + 24 * lane, 24); }
    const u32 u[8] = {code_bytes<0>(cd), code_bytes<3>(cd), code_bytes<6>(cd), code_bytes<9>(cd), code_bytes<12>(cd), code_bytes<15>(cd), code_bytes<18>(cd), code_bytes<21>(cd)};
    for (int idx = 0; idx < 8; idx++) {
      const int s = idx / PER, g = idx % PER, row = kind_v ? v_tok(j, s) : 8 * s + r, group = (kind_v ? 2 * r : 4 * j) + g;
      const u32 word = words[row][group >> 2][(group >> 1) & 1], index = group & 1 ? word >> 16 : word & 0xFFFFu;
      u32 f[4];
      rebuild_pairs(sm[2 * idx], sm[2 * idx + 1], u[idx], index >> 8, base[group], addends[index], f);
      for (int q = 0; q < 4; q++) {                  // elements q and q + 4 of the group
        const int c = kind_v ? 8 * (8 * g + q) + r : 32 * g + 2 * j + (q & 1) + 8 * (q >> 1);
        out[128 * row + c] = (uint16_t)f[q]; out[128 * row + c + (kind_v ? 32 : 16)] = (uint16_t)(f[q] >> 16);
      }
    }
  }
  return raws;
}
