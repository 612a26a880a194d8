// V scaled along d -> MX blocks along the keys, one 32-key block by one warp, and block scales as words of scale atoms: shared by the preparation kernels and by the attention
// kernel that prepares the few tiles of a small call itself.
#pragma once
#include "rk_common.cuh"

namespace rk {

// four floats -> four packed element codes (byte k = code of v[k]); finite inputs only
template <int FMT> RK_DEVINL uint32_t hw_encode4(float a, float b, float c, float d) {
  uint32_t r;
  if (FMT == 0)
    asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\tmov.b32 %0, {lo, hi};\n\t}"
        : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
  else if (FMT == 1)
    asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e5m2x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e5m2x2.f32 hi, %4, %3;\n\tmov.b32 %0, {lo, hi};\n\t}"
        : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
  else if (FMT == 4) {    // two codes per byte, which cross the interfaces one per byte (67 M codes through the integer encoder: 187 us, now 60)
    asm("{\n\t.reg .b8 l, h;\n\tcvt.rn.satfinite.e2m1x2.f32 l, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 h, %4, %3;\n\tmov.b32 %0, {l, h, l, h};\n\t}"
        : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
    r = __byte_perm(r, 0u, 0x4140);
    r = (r | (r << 4)) & 0x0F0F0F0Fu;
  }
  else if (FMT == 2)
    asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e2m3x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e2m3x2.f32 hi, %4, %3;\n\tmov.b32 %0, {lo, hi};\n\t}"
        : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
  else
    asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e3m2x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e3m2x2.f32 hi, %4, %3;\n\tmov.b32 %0, {lo, hi};\n\t}"
        : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}
// Exact value of element code `c` times 2^(s-127) as an fp32.  Normal codes under ordinary scales are
// placed by integer arithmetic (E4M3: bits = (mag + 8 s - 56) << 20); everything else (subnormal codes,
// scale codes near the ends of the range, the other formats) takes the generic multiply.
template <int FMT> RK_DEVINL float decode_scaled(uint32_t c, uint32_t s) {
  if (FMT == 0) {
    const uint32_t mag = c & 0x7Fu;
    if (mag >= 8u && s >= 16u && s <= 240u) return __uint_as_float(((c & 0x80u) << 24) | ((mag + 8u * s - 56u) << 20));
  }
  return decode_elem<FMT>(c) * e8m0_to_f32(s);
}

// The slow form: a thread's NC columns of a block, element by element through fp32; keys k0 .. k0 + 7 are written, and the
// scale codes of NC / 4 columns from c0 on are returned.
template <int FMT, int NC, bool ALL, class PutByte>
__device__ __noinline__ void rebase_slow(const uint8_t* cb, const uint8_t* sb, int n, int k0, int64_t d, int64_t nbd, PutByte put_byte, int c0, uint32_t (&sc)[NC / 4]) {
#pragma unroll 1
  for (int c = 0; c < NC; ++c) {
    float amax = 0.0f, p2 = 1.0f;
    uint32_t code = 0;
    for (int j = 0; j < n; ++j) amax = fmaxf(amax, fabsf(decode_scaled<FMT>(cb[j * d + c], sb[j * nbd])));
    if (amax > 0.0f) block_scale<FMT>(amax, code, p2);
#pragma unroll
    for (int h = 0; h < NC / 4; ++h)
      if (c == c0 + h) sc[h] = code;
    for (int j = k0; j < min(n, k0 + 8); ++j) put_byte(j, c, (uint8_t)encode_rne<FMT>(decode_scaled<FMT>(cb[j * d + c], sb[j * nbd]) * p2));
    if (ALL)
      for (int j = max(n, k0); j < k0 + 8; ++j) put_byte(j, c, 0);
  }
}

// Scales along d, row-major [rows][nbd]: rows i * 32 of a tile from src on (they exist below n), the four blocks of a 128-column chunk (blocks of them exist; src: its first) as
// words of a scale atom, a word per row.  All loads under way at once, as words or halves where they can be (base: where the scales begin).  In the preparation kernels, 6-bit operands:
// d = 64 byte by byte, 8 / 2 heads of 128 keys 13.06 -> 12.84 us a call, 32 / 8 of 640 18.42 -> 18.24; a load after the other, 4-bit, d = 128, 8 / 4 of 256 14.37 -> 14.15, d = 256,
// 16 / 8 of 512 20.37 -> 20.06.
RK_DEVINL void row_scale_words(const uint8_t* src, const uint8_t* base, int64_t nbd, int n, int blocks, uint32_t (&w)[4]) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(base);
  if (((at | nbd) & 3) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = i * 32 < n ? __ldg(reinterpret_cast<const uint32_t*>(src + i * 32 * nbd)) : 0x7F7F7F7Fu;
  } else if (nbd == 2 && (at & 1) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = i * 32 < n ? 0x7F7F0000u | __ldg(reinterpret_cast<const uint16_t*>(src + i * 64)) : 0x7F7F7F7Fu;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t c[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) c[k] = k < blocks && i * 32 < n ? (uint32_t)__ldg(src + i * 32 * nbd + k) : 0x7Fu;
      w[i] = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
    }
  }
}

// Scales along the keys, row-major [key blocks][d]: four adjacent columns of a tile's four key blocks (n_blocks of them exist; in: its first, at the first of the columns) as words of
// a scale atom, a word per column.
RK_DEVINL void key_scale_words(const uint8_t* in, int64_t d, int n_blocks, bool exist, bool aligned, uint32_t (&w)[4]) {
  uint32_t r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    r[k] = 0x7F7F7F7Fu;
    if (exist && k < n_blocks) {
      if (aligned) r[k] = *reinterpret_cast<const uint32_t*>(in + k * d);
      else r[k] = in[k * d] | ((uint32_t)in[k * d + 1] << 8) | ((uint32_t)in[k * d + 2] << 16) | ((uint32_t)in[k * d + 3] << 24);
    }
  }
  const uint32_t a = __byte_perm(r[0], r[1], 0x5140), b = __byte_perm(r[2], r[3], 0x5140), c = __byte_perm(r[0], r[1], 0x7362), e = __byte_perm(r[2], r[3], 0x7362);
  w[0] = __byte_perm(a, b, 0x5410); w[1] = __byte_perm(a, b, 0x7632); w[2] = __byte_perm(c, e, 0x5410); w[3] = __byte_perm(c, e, 0x7632);
}

// ---- V re-blocking: scales along d -> MX blocks along the keys --------------------------------------------------------
// Decode exactly, then the block rule down each column: the same as decoding to fp32 and quantizing again.  The hot form does
// it in f16: a pair of codes goes through the hardware converter, times the row's scale relative to the block's largest, the
// column maxima are packed maxima, the column's factor (a power of two, at least 1) is one more packed product, and the
// pair goes back through the converter.  All of it is exact: values of a format are multiples of 2^-9 (E4M3), 2^-16 (E5M2) or
// 2^-4 (the others) and f16 reaches down to 2^-24, so it holds while the block's scales span no more than kSpan and a column's
// factor stays an f16; other blocks and columns take the slow form through fp32, element by element.
template <int FMT> struct RebaseT { static constexpr int kSpan = FMT == 1 ? 8 : 14; };
// two codes in the low bytes -> packed f16 (exact); an E2M1 code, shifted, is the E2M3 code of its value
template <int FMT> RK_DEVINL uint32_t decode_f16x2(uint32_t codes) {
  uint32_t r;
  if (FMT == 0) asm("{\n\t.reg .b16 c, z;\n\tmov.b32 {c, z}, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, c;\n\t}" : "=r"(r) : "r"(codes));
  else if (FMT == 1) asm("{\n\t.reg .b16 c, z;\n\tmov.b32 {c, z}, %1;\n\tcvt.rn.f16x2.e5m2x2 %0, c;\n\t}" : "=r"(r) : "r"(codes));
  else if (FMT == 3) asm("{\n\t.reg .b16 c, z;\n\tmov.b32 {c, z}, %1;\n\tcvt.rn.f16x2.e3m2x2 %0, c;\n\t}" : "=r"(r) : "r"(codes));
  else asm("{\n\t.reg .b16 c, z;\n\tmov.b32 {c, z}, %1;\n\tcvt.rn.f16x2.e2m3x2 %0, c;\n\t}" : "=r"(r) : "r"(codes));
  return r;
}
// four codes -> two pairs
template <int FMT> RK_DEVINL void decode_f16x4(uint32_t w, uint32_t& lo, uint32_t& hi) {
#define RK_DECODE(T) asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.rn.f16x2." T " %0, l;\n\tcvt.rn.f16x2." T " %1, h;\n\t}" : "=&r"(lo), "=r"(hi) : "r"(w))
  if (FMT == 0) RK_DECODE("e4m3x2"); else if (FMT == 1) RK_DECODE("e5m2x2"); else if (FMT == 3) RK_DECODE("e3m2x2"); else RK_DECODE("e2m3x2");
#undef RK_DECODE
}
// a word of four codes as the converter takes them
template <int FMT> RK_DEVINL uint32_t clean_codes(uint32_t w) {
  return FMT == 4 ? (w & 0x0F0F0F0Fu) << 2 : FMT >= 2 ? w & 0x3F3F3F3Fu : w;
}
RK_DEVINL uint32_t max_u16x2(uint32_t a, uint32_t b) { uint32_t r; asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
RK_DEVINL uint32_t hmul2(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
RK_DEVINL float f16_lo(uint32_t v) { float r; asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tcvt.f32.f16 %0, l;\n\t}" : "=f"(r) : "r"(v)); return r; }
RK_DEVINL float f16_hi(uint32_t v) { float r; asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tcvt.f32.f16 %0, h;\n\t}" : "=f"(r) : "r"(v)); return r; }
// packed f16 pairs -> four codes (finite, exact values: as encode_rne)
template <int FMT> RK_DEVINL uint32_t encode_f16x4(uint32_t lo, uint32_t hi) {
  uint32_t r;
  if (FMT == 0) asm("{\n\t.reg .b16 a, b;\n\tcvt.rn.satfinite.e4m3x2.f16x2 a, %1;\n\tcvt.rn.satfinite.e4m3x2.f16x2 b, %2;\n\tmov.b32 %0, {a, b};\n\t}" : "=r"(r) : "r"(lo), "r"(hi));
  else if (FMT == 1) asm("{\n\t.reg .b16 a, b;\n\tcvt.rn.satfinite.e5m2x2.f16x2 a, %1;\n\tcvt.rn.satfinite.e5m2x2.f16x2 b, %2;\n\tmov.b32 %0, {a, b};\n\t}" : "=r"(r) : "r"(lo), "r"(hi));
  else r = hw_encode4<FMT>(f16_lo(lo), f16_hi(lo), f16_lo(hi), f16_hi(hi));
  return r;
}

// One warp's 32 keys x 8 NC columns (unit cu of them): codes and scales are those of the block's first key, n keys exist.  A lane has keys k0 = 8 (lane / 8) to k0 + 7 and NC
// adjacent columns; put(key, words) takes its codes of a key, put_byte(key, column of its NC, code) one of them in the slow form.  ALL: put is called for keys that do
// not exist as well, with zeros.  sc: the new scale codes of columns NC (lane % 8) + (NC / 4) (lane / 8) + 0 .. of the unit.  fac_sm: scratch of this warp.
// Idx: of an element within the 32 rows of d columns; int where d <= INT_MAX / 32, as in the attention calls.
template <int FMT, int NC, bool ALL, class Idx, class Put, class PutByte>
RK_DEVINL void rebase_block(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ scales, Idx d, Idx cu, int n, uint32_t (*fac_sm)[32], int lane, Put put,
                            PutByte put_byte, uint32_t (&sc)[NC / 4]) {
  constexpr int NW = NC / 4, NB = NC / 4, CP = NC / 4;             // words per key of a thread; 32-column blocks of a warp; columns of a lane's quarter
  const int k0 = (lane >> 3) * 8, b = (lane & 7) * NC / 32;
  const Idx nbd = d >> 5, col = cu * 8 * NC + (lane & 7) * NC;
  const bool in = col < d && n > 0;
  const uint8_t* src = codes + col;
  const uint8_t* const src0 = src + k0 * d;
  const int rows = in ? n - k0 : 0;                              // of this lane's eight
  uint32_t w[8][NW];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const bool live = i < rows;
    const uint8_t* q = src0 + i * d;
    if (NC == 8) {
      const uint2 v = live ? __ldg(reinterpret_cast<const uint2*>(q)) : make_uint2(0u, 0u);
      w[i][0] = v.x; w[i][NW - 1] = v.y;
    } else {
      w[i][0] = live ? __ldg(reinterpret_cast<const uint32_t*>(q)) : 0u;
    }
  }
  // the rows' scales relative to the block's largest, as packed f16; lane = key
  int smax = 0;
  bool hot = true;
  const uint8_t* sk = scales + lane * nbd + cu * NB;
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    const bool live = lane < n && cu * NB + c < nbd;
    const int s = live ? (int)__ldg(sk + c) : -1;
    const int top = __reduce_max_sync(0xffffffffu, s), low = __reduce_min_sync(0xffffffffu, live ? s : 255);
    fac_sm[c][lane] = live ? (uint32_t)max(15 + s - top, 1) * 0x04000400u : 0u;
    if (c == b) { smax = max(top, 0); hot = low >= 20 && top <= 235 && top - low <= RebaseT<FMT>::kSpan; }
  }
  __syncwarp();
  uint32_t m[2 * NW];                                            // maxima of column pairs
#pragma unroll
  for (int i = 0; i < 2 * NW; ++i) m[i] = 0u;
  uint32_t x[8][2 * NW];
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    const uint4 f4 = *reinterpret_cast<const uint4*>(&fac_sm[b][k0 + i]);
    const uint32_t f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int e = 0; e < 4; e += 2)
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        uint32_t c[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          decode_f16x4<FMT>(clean_codes<FMT>(w[i + e + h][q]), c[h][0], c[h][1]);
          x[i + e + h][2 * q] = hmul2(c[h][0], f[e + h]);
          x[i + e + h][2 * q + 1] = hmul2(c[h][1], f[e + h]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
          m[2 * q + h] = __vimax3_u16x2(m[2 * q + h], x[i + e][2 * q + h] & 0x7FFF7FFFu, x[i + e + 1][2 * q + h] & 0x7FFF7FFFu);
      }
  }
  __syncwarp();                                                  // fac_sm has been read
  // The four lanes of a column group end up with the maxima of a quarter of its columns each, work out those scales and
  // hand the factors back.
  const bool h16 = lane & 16, h8 = lane & 8;
  uint32_t mine;
  if (NC == 8) {
    const uint32_t a = max_u16x2(h16 ? m[NW] : m[0], __shfl_xor_sync(0xffffffffu, h16 ? m[0] : m[NW], 16));
    const uint32_t c = max_u16x2(h16 ? m[2 * NW - 1] : m[1], __shfl_xor_sync(0xffffffffu, h16 ? m[1] : m[2 * NW - 1], 16));
    mine = max_u16x2(h8 ? c : a, __shfl_xor_sync(0xffffffffu, h8 ? a : c, 8));
  } else {
    mine = max_u16x2(h16 ? m[1] : m[0], __shfl_xor_sync(0xffffffffu, h16 ? m[0] : m[1], 16));
    mine = max_u16x2(mine, __shfl_xor_sync(0xffffffffu, mine, 8));
    if (h8) mine >>= 16;
  }
  const float unit = __uint_as_float((uint32_t)smax << 23);      // 2^(smax - 127)
  uint32_t fac = 0u, f[2 * NW];
#pragma unroll
  for (int h = 0; h < CP; ++h) {
    const float am = (h ? f16_hi(mine) : f16_lo(mine)) * unit;
    uint32_t code = 0; float p2;
    int up = 0;                                                  // log2 of the column's factor
    if (am > 0.0f) { block_scale<FMT>(am, code, p2); up = (int)(__float_as_uint(p2) >> 23) - 254 + smax; }
    hot = hot && up <= 15 && (FMT > 1 || am < __int_as_float(0x7f800000));        // (NaN and infinity encodings are numbers here)
    sc[h] = in ? code : 0x7Fu;                                   // of columns and key blocks that do not exist: 2^0
    fac |= (uint32_t)((15 + up) & 31) << (10 + 16 * h);
  }
  hot = (__ballot_sync(0xffffffffu, !hot) & (0x01010101u << (lane & 7))) == 0u;
#pragma unroll
  for (int i = 0; i < 2 * NW; ++i) {
    f[i] = __shfl_sync(0xffffffffu, fac, (lane & 7) + (NC == 8 ? 8 * i : 16 * i));
    if (NC == 4) f[i] |= __shfl_sync(0xffffffffu, fac, (lane & 7) + 16 * i + 8) << 16;
  }
  if (col < d) {
    if (hot || n == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (!ALL && k0 + i >= n) break;
        uint32_t o[NW];
#pragma unroll
        for (int q = 0; q < NW; ++q) o[q] = encode_f16x4<FMT>(hmul2(x[i][2 * q], f[2 * q]), hmul2(x[i][2 * q + 1], f[2 * q + 1]));
        put(k0 + i, o);
      }
    } else {
      rebase_slow<FMT, NC, ALL>(src, scales + col / 32, n, k0, d, nbd, put_byte, (lane >> 3) * CP, sc);
    }
  }
}

}  // namespace rk
