// Split-KV decode attention over an MXFP8 KV cache on the 5th-generation tensor cores.
//
// Same semantics as rk_decode.cu (prefill at S_q = 1, GQA head map
// kernels/flash_attention_mx_gqa/kernel.cpp:109-115; K and V decoded exactly, fp32 softmax state, no P
// requant in the reference sense), but the raw E4M3 bytes of K and V go from shared memory straight into
// tcgen05 block-scaled MMAs, so no thread ever converts a cache byte:
//
//   S^T[key][n]   = K_tile[128 keys x 128 d] . Qterms^T          A = K tile as TMA wrote it (K-major, SW128),
//                                                                scale-factor A = the tile's E8M0 key scales,
//                                                                B = the query heads as 2 MXFP8 terms each
//                                                                (q = hi + lo exactly: bf16 has 8 significant
//                                                                bits, an E4M3 term 4), N = 16
//   O^T[d][n]    += V_tile^T[128 d x 128 keys] . Pterms          A = V tile as TMA wrote it (MN-major), unit
//                                                                scales; B = P (MN-major: a key's codes side by
//                                                                side), per (32-column group q of d, term, head):
//                                                                p * 2^(sv[key][q]) as 2 MXFP8 terms with one E8M0
//                                                                scale per 32 keys, N = 8 HH
//
// V's scale belongs to (key, 32-column group of d); a block-scaled MMA has one scale per (row, 32 keys), so the scale is
// folded into P: column (q, term, h) of B carries p[h][key] * 2^(sv[key][q] - svmax[q]), and its block scale carries
// svmax[q] (the largest V scale among the block's 32 keys) and the exponent of the block's largest p.  A power of two
// moves an E4M3 code by 8 per step, so a key's p is converted once per head and the four groups' codes are byte
// subtractions on packed words (where the V scales of a block lie more than kFarOctaves apart: once per head and group).  Row d of O^T only uses the columns of its own group q = d / 32.
//
// One CTA per SM, and the CTAs share the key tiles of the whole call evenly: the tiles of all sequences in a row (each
// sequence as long as it is) are cut into as many equal ranges as there are CTAs.  A range is a list of segments, each a
// run of tiles of one (batch, KV head) unit; a unit that lies in one range is finished here, one that crosses ranges leaves
// partials for the combine kernel.  (One split count for all sequences lets the longest ones set the time.)
//
// A tile is a serial chain -- S from TMEM, maximum, exponentials, P in shared memory, P V -- several times as long as its
// bytes take to arrive, so four groups of four worker warps each take every fourth tile.  One warp loads, one puts the
// tiles' key scales into the order of a scale atom, one issues S = K Q^T, one O += V^T P (with the scales in the issuer a
// tile took it 1100 cycles, as long as HBM), one prepares the query terms of the next segment (loading and quantizing eight
// heads takes longer than a tile, so in another warp's stream it held back every short sequence).
//   worker warp w: group w / 4, thread = key (w % 4) * 32 + lane of the tile for S and P, and column d of O^T.
// p, O and the row sums are relative to a reference m_ref per head (and to one V scale per group of 32 columns): the first
// tile's maximum, handed from tile to tile, and replaced by a tile's own maximum where that is more than 2^8 above it (V scales:
// 2^32), so O is rescaled about never.  The p of the key that set the reference is 1, which two terms hold exactly: with the
// weight on few keys it is the error of the largest p that counts.  (References that are integers, so that the codes need not
// wait for the other warps' maxima, leave that p with the rounding of any other: errors of 5.9e-4 of the result instead of
// 5.2e-4 with queries of four times unit variance, 5.8e-4 instead of 4.1e-4 with twelve times.)  A warp's block scale carries
// the power of two of the largest p of its 32 keys.
// A segment ends in the group of its last tile alone: it reads O (one of four accumulators, used in turn) and the row sums
// the other warps left, while those are in the next segment's tiles.  (With a meeting of all workers at its end a segment
// cost 5000 cycles, four tiles' time.)
//
// Included by rk_decode.cu (one translation unit: both kernels share the launcher).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "rk_common.cuh"
#include "rk_internal.h"

namespace rk {

namespace dtc {
constexpr int kGroups = 4;                        // worker groups of four warps
constexpr int kWorkers = 4 * kGroups;             // worker warps
constexpr int kWarpTma = kWorkers, kWarpSf = kWorkers + 1, kWarpQk = kWorkers + 2, kWarpPv = kWorkers + 3,
              kWarpQ = kWorkers + 4;
constexpr int kThreads = (kWorkers + 5) * 32;
constexpr int kTile = 128;                        // keys per stage
constexpr int kD = 128;
constexpr int kMaxGrp = 8;                        // query heads per KV head this kernel handles
constexpr int kNq = 16;                           // B rows of the QK^T MMA: term * HH + h (rows past 2 HH stay zero)
constexpr int kTileBytes = kTile * kD;            // 16384
constexpr int kStageBytes = 2 * kTileBytes + 2 * 512;   // K, V, K scales [128][4], V scales [128][4]
constexpr int kOBufs = 4, kRing = 8;              // accumulators in turn; tiles whose references are kept
constexpr uint32_t kFarOctaves = 4;               // V scales further below their block's largest are not taken by moving codes
constexpr float kBump = 8.0f, kBumpV = 32.0f;     // rescale O when a maximum (a V scale) passes its reference by more than 2^this

// Per head capacity HH (4 or 8): column n of the PV MMA = q * 2 HH + term * HH + h.
template <int HH> struct Lay {
  static constexpr int kNp = 8 * HH;
  static constexpr int kStages = 5;
  // P tiles: rows of 128 bytes (128-byte swizzle), one row per key; a group's tile takes kNp bytes of each row
  static constexpr int kPerAtom = 128 / kNp;
  static constexpr int kPBytes = kGroups / kPerAtom * kTileBytes;
  // shared-memory map (offsets from a 1024-byte aligned base)
  static constexpr int stage_off = 0;
  static constexpr int p_off = kStages * kStageBytes;
  static constexpr int q_off = p_off + kPBytes;                // [2 segments][16 rows][128 B], K-major SW128
  static constexpr int sfp_off = q_off + 2 * 2048;             // a 512-byte scale atom of P per group
  static constexpr int sfq_off = sfp_off + kGroups * 512;      // scale atoms of the query terms, [2 segments]
  static constexpr int one_off = sfq_off + 2 * 512;            // scale atom of ones (code 127) for V
  static constexpr int xchg_off = one_off + 512;               // [groups][2][4 warps][16] floats: maxima of the heads, then svmax
  static constexpr int ring_off = xchg_off + kGroups * 2 * 4 * 16 * 4;  // [8 tiles][16] floats: references after a tile, same order
  static constexpr int ref_off = ring_off + kRing * 16 * 4;    // [16 warps][16] floats: the references a warp's sums are relative to
  static constexpr int seg_off = ref_off + kWorkers * 16 * 4;  // end of a segment: [kOBufs][16 warps][8] float2: sum, its reference
  static constexpr int bar_off = seg_off + kOBufs * kWorkers * 8 * 8;
  static constexpr int bFull = 0, bEmpty = bFull + kStages, bSF = bEmpty + kStages, bSE = bSF + kGroups, bPF = bSE + kGroups,
                       bMX = bPF + kGroups, bPV = bMX + kGroups, bKS = bPV + kGroups, bQF = bKS + kStages, bQE = bQF + 2, bRef = bQE + 2,
                       bSL = bRef + kRing, bOE = bSL + kOBufs, bDrain = bOE + kOBufs,
                       nBars = bDrain + 2;
  static constexpr int misc_off = bar_off + nBars * 8;         // tmem base, abort flag
  static constexpr int total = misc_off + 16;
  static_assert(kStageBytes % 1024 == 0 && p_off % 1024 == 0 && q_off % 1024 == 0, "swizzled tiles need 1024-byte alignment");
  static_assert(total + 1024 <= 232448, "shared memory of a CTA");
};

// TMEM columns
constexpr uint32_t cS = 0;                        // 16 per group
constexpr uint32_t cO = 64;                       // up to 64 per accumulator
constexpr uint32_t cSfK = 320;                    // 4 per stage
constexpr uint32_t cSfQ = 344;                    // 4 per segment parity
constexpr uint32_t cSfP = 352;                    // 4 per group
constexpr uint32_t cSfOne = 368;
constexpr uint32_t kTmemCols = 512;
}  // namespace dtc

struct DecodeTcParams {
  const __nv_bfloat16* q;
  const uint8_t* k_scale;
  const uint8_t* v_scale;
  const int32_t* kv_len;
  __nv_bfloat16* o;
  float* lse;
  float* part_o;    // nsplit > 0: [B*H][nsplit][128]; 0: [CTA][2][grp][128] -- a CTA leaves at most two partials, of the unit its
                    // range begins inside of (slot 0) and of the one its range ends inside of (slot 1)
  float* part_ml;   // the same indices, [2]: reference maximum in the log2 domain, l
  int* status;
  int B, H, H_kv, L, grp, nsplit;                 // nsplit: the caller's split count per unit, or 0 for equal ranges
  float scale_log2;
};

RK_DEVINL int dtc_len(const DecodeTcParams& p, int b) { return p.kv_len ? min(max(p.kv_len[b], 0), p.L) : p.L; }
// 1 / l and the log-sum-exp.  l is 0 without keys; a NaN score makes it NaN and must reach every column of O: the codes of a NaN p
// that were moved down are numbers.
RK_DEVINL float dtc_inverse(float l) { return l == 0.0f ? 1.0f : 1.0f / l; }
RK_DEVINL float dtc_lse(float m, float l) { return l == 0.0f ? __int_as_float(0xff800000) : m * 0.6931471805599453f + logf(l); }
RK_DEVINL int dtc_tiles(int len) { return (len + dtc::kTile - 1) / dtc::kTile; }
// first tile of CTA c of g when t tiles are shared evenly
RK_DEVINL int dtc_first(int t, int c, int g) {
  const uint32_t q = (uint32_t)t / (uint32_t)g, r = (uint32_t)t - q * (uint32_t)g;      // t c / g without a 64-bit division (g < 2^16)
  return (int)(q * (uint32_t)c + r * (uint32_t)c / (uint32_t)g);
}

// Ranges that t tiles are cut into for g CTAs: as many as there are tiles at most, so that none is empty and the CTAs without one are the last (one sequence of
// 1000 keys 11.4 -> 10.4 us, of 200 10.4 -> 9.7, against empty ranges between the others, which the combine kernel then has to tell apart).  Ranges of two tiles
// at least: 10.6 and 9.2, but 8 heads of 128 keys 8.3 -> 9.1 and short sequences of several heads 3-4 % slower; of four 11.1 and 10.5.
RK_DEVINL int dtc_ranges(int t, int g) { return min(g, max(1, t)); }

// The segments of a CTA's range of tiles, in order.  Every warp walks its own copy.
struct DtcSegments {
  int b, hkv, t0, n;        // current segment: tiles t0 .. t0 + n - 1 of unit (b, hkv)
  int len, n_unit;          // keys and tiles of the unit
  int left;                 // tiles of the range from this segment on; 0 = done

  RK_DEVINL void clip() { n = min(n_unit - t0, left); }
  RK_DEVINL void seek(const DecodeTcParams& p) { len = dtc_len(p, b); n_unit = dtc_tiles(len); }
  RK_DEVINL void next(const DecodeTcParams& p) {
    left -= n;
    t0 = 0;
    if (left <= 0) return;
    if (++hkv == p.H_kv) {
      hkv = 0;
      do { ++b; seek(p); } while (n_unit == 0);
    }
    clip();
  }
  RK_DEVINL void start(const DecodeTcParams& p, int lane) {      // whole warp
    int total = 0, first;                                        // tiles of the whole call; the CTA's first of them
    if (p.nsplit > 0) {
      const int split = blockIdx.x % p.nsplit, u = blockIdx.x / p.nsplit;
      b = u / p.H_kv; hkv = u % p.H_kv;
      seek(p);
      const int per = (n_unit + p.nsplit - 1) / p.nsplit;
      t0 = split * per;
      left = max(0, min(n_unit, t0 + per) - t0);
      clip();
      return;
    }
    if (!p.kv_len) {
      n_unit = dtc_tiles(p.L); len = p.L;
      total = p.B * p.H_kv * n_unit;
      const int g = dtc_ranges(total, gridDim.x);
      const int c = min((int)blockIdx.x, g);
      first = dtc_first(total, c, g);
      left = c < g ? dtc_first(total, c + 1, g) - first : 0;
      if (left <= 0) { b = hkv = t0 = n = 0; return; }
      const int u = first / n_unit;
      b = u / p.H_kv; hkv = u % p.H_kv; t0 = first - u * n_unit;
      clip();
      return;
    }
    const int len0 = lane < p.B ? dtc_len(p, lane) : 0;           // the first 32 lengths are read once (a load is 0.4 us here)
    const int tiles0 = dtc_tiles(len0);
    int incl0 = tiles0;                                            // of those, up to and with this lane's; their total comes with it (a reduction of its own: 0.15 us a call)
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) { const int o = __shfl_up_sync(0xffffffffu, incl0, s); if (lane >= s) incl0 += o; }
    if (p.B > 32) {
      for (int i = lane + 32; i < p.B; i += 32) total += dtc_tiles(dtc_len(p, i));
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) total += __shfl_xor_sync(0xffffffffu, total, s);
    }
    total += __shfl_sync(0xffffffffu, incl0, 31);
    total *= p.H_kv;
    const int g = dtc_ranges(total, gridDim.x), c = min((int)blockIdx.x, g);
    first = dtc_first(total, c, g);
    left = c < g ? dtc_first(total, c + 1, g) - first : 0;
    b = hkv = t0 = n = n_unit = len = 0;
    if (left <= 0) return;
    int base = 0;                                              // tiles of the sequences before this block of 32
    for (int i0 = 0;; i0 += 32) {
      const int my_len = i0 == 0 ? len0 : i0 + lane < p.B ? dtc_len(p, i0 + lane) : 0;
      const int mine = (i0 == 0 ? tiles0 : dtc_tiles(my_len)) * p.H_kv;
      int incl = incl0 * p.H_kv;
      if (i0 > 0) {
        incl = mine;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) { const int o = __shfl_up_sync(0xffffffffu, incl, s); if (lane >= s) incl += o; }
      }
      const uint32_t past = __ballot_sync(0xffffffffu, base + incl > first);
      if (past) {
        const int w = __ffs(past) - 1;
        b = i0 + w;
        const int off = first - base - __shfl_sync(0xffffffffu, incl - mine, w);
        len = __shfl_sync(0xffffffffu, my_len, w);
        n_unit = dtc_tiles(len);
        hkv = off / n_unit; t0 = off - hkv * n_unit;
        clip();
        return;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
};

// two fp32 -> two E4M3 codes, RNE, saturating: bits 15:8 = code(hi), bits 7:0 = code(lo)
RK_DEVINL uint32_t cvt_e4m3x2(float hi, float lo) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
// the two codes back to fp32 (exact)
RK_DEVINL void e4m3x2_to_f32(uint32_t codes, float& hi, float& lo) {
  uint32_t h2;
  asm("{\n\t.reg .b16 c;\n\tcvt.u16.u32 c, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, c;\n\t}" : "=r"(h2) : "r"(codes));
  const __half2 v = *reinterpret_cast<const __half2*>(&h2);
  lo = __low2float(v);
  hi = __high2float(v);
}
RK_DEVINL uint32_t redux_max_u32(uint32_t v) {
  uint32_t r;
  asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
  return r;
}
// byte offset of (row n, byte x) in a K-major tile with 128-byte rows and the 128-byte swizzle
RK_DEVINL int sw128(int n, int x) { return n * 128 + ((((x >> 4) ^ (n & 7))) << 4) + (x & 15); }

// 2^e as fp32 for an integer e; below the normal range the result is 0, above it the largest power of two
RK_DEVINL float pow2i(int e) {
  const int f = e + 127;
  return __uint_as_float(f <= 0 ? 0u : ((uint32_t)(f > 254 ? 254 : f) << 23));
}

// maximum over the warp (NaNs lose)
RK_DEVINL float redux_max_f32(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
// The bounded wait of the kernel's loops, in its short form (the code of a tile runs cold at the start of every launch, and a
// short sequence is over before it is warm).  False, with the code recorded, when it gave up.
RK_DEVINL bool dtc_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (__builtin_expect(mbar_wait_lean(bar, parity, abort_flag), 1)) return true;
  report_wait_failure(abort_flag, status, code);
  return false;
}
// bit 7 of every byte that is at least N (1 .. 128)
template <uint32_t N> RK_DEVINL uint32_t bytes_at_least(uint32_t w) { return (((w & 0x7F7F7F7Fu) + (128u - N) * 0x01010101u) | w) & 0x80808080u; }
// p = hi + lo / 16 in E4M3, two heads at a time: bits 15:8 of the codes = p1, bits 7:0 = p0
RK_DEVINL void p_terms(float p1, float p0, uint32_t& hi, uint32_t& lo) {
  hi = cvt_e4m3x2(p1, p0);
  float a1, a0;
  e4m3x2_to_f32(hi, a1, a0);
  lo = cvt_e4m3x2((p1 - a1) * 16.0f, (p0 - a0) * 16.0f);
}
// Four packed E4M3 codes divided by 2^(d / 8): d8 = d in every byte, d a multiple of 8 up to 120.  Codes that leave the
// normal range become 0 (or lose their hidden bit), an absolute error of 2^-15 of the block's largest element.  SIGN: codes
// may be negative.
template <bool SIGN> RK_DEVINL uint32_t e4m3x4_down(uint32_t w, uint32_t d8) {
  const uint32_t r = (w | 0x80808080u) - d8, m = r & 0x80808080u;       // bit 7 is left where the magnitude was at least d
  const uint32_t mag = r & (m - (m >> 7));
  return SIGN ? mag | (w & 0x80808080u) : mag;
}

// A worker warp: thread = key kt of a tile (S, P) and column d = kt (O).
template <int HH>
RK_DEVINL void decode_tc_worker(const DecodeTcParams& p, uint8_t* smem, uint64_t* bars, uint32_t tmem_base, volatile int* abort_flag,
                                DtcSegments& seg, int warp, int lane) {
  using namespace dtc;
  using L = Lay<HH>;
  constexpr int kStages = L::kStages;
  const float NEG_INF = __int_as_float(0xff800000);
  const int g = warp >> 2, wq = warp & 3, kt = wq * 32 + lane;
  const uint32_t lane_addr = ((uint32_t)(wq * 32)) << 16;
  const uint32_t s_addr = tmem_base + lane_addr + cS + g * 16;
  const uint32_t o_row = tmem_base + lane_addr + cO + wq * 2 * HH;               // row d = kt: only the columns of its q = wq count
  // this key's row of the group's P tile; 16-byte chunk i of it sits at (chunk0 + i) ^ (kt & 7)
  uint8_t* prow = smem + L::p_off + (g / L::kPerAtom) * kTileBytes + kt * 128;
  const int chunk0 = (g % L::kPerAtom) * (L::kNp / 16);
  float* xchg = reinterpret_cast<float*>(smem + L::xchg_off) + g * 128;          // [2][4 warps][16]
  float* ring = reinterpret_cast<float*>(smem + L::ring_off);                    // [kRing][16]
  float* ref = reinterpret_cast<float*>(smem + L::ref_off) + warp * 16;          // what this warp's sums are relative to
  float2* sums = reinterpret_cast<float2*>(smem + L::seg_off);                   // [kOBufs][16 warps][8]
  const int item = lane & 15;                                                    // 0..7: a head, 8..11: a group of 32 columns of d
  bool ok = true;
  int j0 = 0;                                                                    // tiles of this CTA before the segment

  for (int sg = 0; seg.left > 0 && ok; ++sg, j0 += seg.n, seg.next(p)) {
    const uint32_t o_addr = o_row + (sg % kOBufs) * 64;
    float l_part[HH];
#pragma unroll
    for (int h = 0; h < HH; ++h) l_part[h] = 0.0f;
    float ref_item = 0.0f;                                                       // of this lane's item, as in ref[]
    const int i_first = (g - j0) & (kGroups - 1);

    for (int i = i_first; i < seg.n; i += kGroups) {
      const int j = j0 + i, st = j % kStages, par = (j / kGroups) & 1;
      uint8_t* sb = smem + L::stage_off + st * kStageBytes;
      ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bSF + g], par, abort_flag, p.status, 501));
      if (!ok) break;
      tc_fence_after();
      uint32_t c[2 * HH];
      if (HH == 8) tmem_ld16(s_addr, c); else tmem_ld8(s_addr, c);
      uint32_t svw = *reinterpret_cast<const uint32_t*>(sb + 2 * kTileBytes + 512 + kt * 4);
      tc_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[L::bSE + g]);

      // ---- scores, the warp's maxima ----------------------------------------------------------------------------
      float s[HH];
#pragma unroll
      for (int h = 0; h < HH; ++h) s[h] = (__uint_as_float(c[h]) + __uint_as_float(c[HH + h])) * p.scale_log2;   // log2 domain
      const bool tail = (seg.t0 + i + 1) * kTile > seg.len;
      const bool valid = (seg.t0 + i) * kTile + kt < seg.len;
      if (tail && !valid) {
#pragma unroll
        for (int h = 0; h < HH; ++h) s[h] = NEG_INF;
        svw = 0u;
      }
      uint32_t svmax[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) svmax[q] = redux_max_u32((svw >> (8 * q)) & 0xFFu);
      float* xw = xchg + par * 64 + wq * 16;
#pragma unroll
      for (int h = 0; h < HH; h += 4) {
        const float4 m = make_float4(redux_max_f32(s[h]), redux_max_f32(s[h + 1]), redux_max_f32(s[h + 2]), redux_max_f32(s[h + 3]));
        if (lane == 0) *reinterpret_cast<float4*>(xw + h) = m;
      }
      if (lane == 0) {
        *reinterpret_cast<float4*>(xw + 8) = make_float4((float)svmax[0], (float)svmax[1], (float)svmax[2], (float)svmax[3]);
        mbar_arrive(&bars[L::bMX + g]);
      }

      // octaves from each V scale to its block's largest; is one far (scale code 0 is a block of zeros)?
      const uint32_t dw = (svmax[0] | (svmax[1] << 8) | (svmax[2] << 16) | (svmax[3] << 24)) - svw;
      const bool far = __any_sync(0xffffffffu, (bytes_at_least<kFarOctaves + 1>(dw) & bytes_at_least<1>(svw)) != 0u);

      // ---- references ---------------------------------------------------------------------------------------------
      ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bMX + g], par, abort_flag, p.status, 504) &&
                                       (i == 0 || dtc_wait(&bars[L::bRef + (j - 1) % kRing], ((j - 1) / kRing) & 1, abort_flag, p.status, 507)));
      if (!ok) break;
      {
        const float* xr = xchg + par * 64 + (lane >> 4) * 32 + item;
        float top = fmaxf(xr[0], xr[16]);
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
        top = fmaxf(top, -1.0e30f);
        const float before = i == 0 ? top : ring[((j - 1) % kRing) * 16 + item];
        // every warp of the group sees the same maxima and references, so what follows is uniform over the group
        const float now = top > before + (item < 8 ? kBump : kBumpV) ? top : before;
        if (wq == 0) {
          if (lane < 16) ring[(j % kRing) * 16 + lane] = now;
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[L::bRef + j % kRing]);
        }
        if (i == i_first || __any_sync(0xffffffffu, now != ref_item)) {
          if (__any_sync(0xffffffffu, now != before)) {
            // rescale this thread's row of O once the tile before has been added; its own P V comes after this
            ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bPV + ((j - 1) & (kGroups - 1))], ((j - 1) / kGroups) & 1, abort_flag, p.status, 502));
            if (!ok) break;
            tc_fence_after();
            uint32_t o[2 * HH];
            if (HH == 8) tmem_ld16(o_addr, o); else tmem_ld8(o_addr, o);
            tc_wait_ld();
            const float down = before - now, down_v = __shfl_sync(0xffffffffu, down, 8 + wq);
#pragma unroll
            for (int h = 0; h < HH; ++h) {
              const float f = ex2_approx(fmaxf(__shfl_sync(0xffffffffu, down, h) + down_v, -126.0f));
              o[h] = __float_as_uint(__uint_as_float(o[h]) * f);
              o[HH + h] = __float_as_uint(__uint_as_float(o[HH + h]) * f);
            }
            if (HH == 8) tmem_st16(o_addr, o); else tmem_st8(o_addr, o);
            tc_wait_st();
          }
          // first tile of the segment here, or a reference moved here or in another group: this warp's sums follow
          if (i != i_first) {
            const float down = ref_item - now;
#pragma unroll
            for (int h = 0; h < HH; ++h) l_part[h] *= ex2_approx(__shfl_sync(0xffffffffu, down, h));
          }
          ref_item = now;
          __syncwarp();
          if (lane < 16) ref[lane] = now;
          __syncwarp();
        }
      }
      // ---- p = 2^(s - m_ref), scaled into [2^7, 2^8) by the warp's largest, in two terms; a word holds the codes of four heads ----
      // (s is rounded before m_ref is taken off: with one rounding for both, as fmaf has, the largest p of scores beyond 2^24
      // would not be 1.)
      // Steps from the references to this warp's own maxima: heads at most 9, V scales at most 32; far below, the product vanishes.
      const int eh = max((int)(__float_as_uint(ex2_approx(xw[item] - ref_item)) >> 23), 7);
      const int step = item < 8 ? eh - 126 : __float2int_rn(fmaxf(xw[item] - ref_item, -200.0f));
      const int step_h = __shfl_sync(0xffffffffu, step, lane & (HH - 1));
      const float scale_up = __uint_as_float((uint32_t)(261 - eh) << 23);              // 2^(8 - step)
      uint32_t hi[HH / 4], lo[HH / 4];
#pragma unroll
      for (int h = 0; h < HH; h += 4) {
        const float4 m4 = *reinterpret_cast<const float4*>(ref + h);
        const float m[4] = {m4.x, m4.y, m4.z, m4.w};
        uint32_t ch[2], cl[2];
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          float &p0 = s[h + e], &p1 = s[h + e + 1];
          p0 = ex2_approx(p0 - m[e]);                              // masked keys give 0
          p1 = ex2_approx(p1 - m[e + 1]);
          l_part[h + e] += p0;
          l_part[h + e + 1] += p1;
          p0 *= __shfl_sync(0xffffffffu, scale_up, h + e);
          p1 *= __shfl_sync(0xffffffffu, scale_up, h + e + 1);
          p_terms(p1, p0, ch[e / 2], cl[e / 2]);
        }
        hi[h / 4] = __byte_perm(ch[0], ch[1], 0x5410);
        lo[h / 4] = __byte_perm(cl[0], cl[1], 0x5410);
      }
      // the P tile is free once the P V that read it (the group's previous tile) has completed
      if (j >= kGroups) {
        ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bPV + g], par ^ 1, abort_flag, p.status, 503));
        if (!ok) break;
      }
      // A code moved down loses what falls below the normal range, 2^-15 of the block's largest element: nothing while the V scales
      // of its keys lie close together, but all of a heavy key whose scale lies far below that of a light one.  Blocks with
      // such keys are converted again for every group of columns, which rounds into the subnormals.
      if (__builtin_expect(!far, 1)) {
        uint32_t d8[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) d8[q] = min((dw >> (8 * q)) & 0xFFu, 15u) * 0x08080808u;
        if (HH == 8) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<uint4*>(prow + (((chunk0 + q) ^ (kt & 7)) << 4)) =
                make_uint4(e4m3x4_down<false>(hi[0], d8[q]), e4m3x4_down<false>(hi[HH / 4 - 1], d8[q]),
                           e4m3x4_down<true>(lo[0], d8[q]), e4m3x4_down<true>(lo[HH / 4 - 1], d8[q]));
        } else {
#pragma unroll
          for (int q = 0; q < 4; q += 2)
            *reinterpret_cast<uint4*>(prow + (((chunk0 + q / 2) ^ (kt & 7)) << 4)) =
                make_uint4(e4m3x4_down<false>(hi[0], d8[q]), e4m3x4_down<true>(lo[0], d8[q]),
                           e4m3x4_down<false>(hi[0], d8[q + 1]), e4m3x4_down<true>(lo[0], d8[q + 1]));
        }
      } else {
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          const float f = __uint_as_float((127u - min((dw >> (8 * q)) & 0xFFu, 127u)) << 23);
          uint32_t w[2 * HH / 4];                                   // hi words, then lo words
#pragma unroll
          for (int h = 0; h < HH; h += 4) {
            uint32_t ch[2], cl[2];
            p_terms(s[h + 1] * f, s[h] * f, ch[0], cl[0]);
            p_terms(s[h + 3] * f, s[h + 2] * f, ch[1], cl[1]);
            w[h / 4] = __byte_perm(ch[0], ch[1], 0x5410);
            w[HH / 4 + h / 4] = __byte_perm(cl[0], cl[1], 0x5410);
          }
          if (HH == 8) *reinterpret_cast<uint4*>(prow + (((chunk0 + q) ^ (kt & 7)) << 4)) = make_uint4(w[0], w[1], w[HH / 4], w[2 * HH / 4 - 1]);
          else *reinterpret_cast<uint2*>(prow + (((chunk0 + q / 2) ^ (kt & 7)) << 4) + (q & 1) * 8) = make_uint2(w[0], w[HH / 4]);
        }
      }
      if (__builtin_expect(tail && !valid, 0)) {   // a key past kv_len: its V row may hold anything; 0 * NaN must not reach the accumulator
        uint4* vrow = reinterpret_cast<uint4*>(sb + kTileBytes + kt * 128);
#pragma unroll
        for (int q = 0; q < 8; ++q) vrow[q] = make_uint4(0u, 0u, 0u, 0u);
      }

#pragma unroll
      for (int part = 0; part < L::kNp / 32; ++part) {          // block scale of column n for this warp's 32 keys (k-block = wq)
        const int n = part * 32 + lane, q = n / (2 * HH), term = (n / HH) & 1;
        const int code = min(max(127 + step_h + __shfl_sync(0xffffffffu, step, 8 + q), 5), 254) - 4 * term;
        smem[L::sfp_off + g * 512 + lane * 16 + part * 4 + wq] = (uint8_t)code;
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[L::bPF + g]);
    }
    if (!ok) break;

    // ---- end of the segment: every warp leaves its row sums; the group of the last tile puts the result together --------
    const int ob = sg % kOBufs;
    if (sg >= kOBufs) {                                            // the slot has been read
      ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bOE + ob], (sg / kOBufs - 1) & 1, abort_flag, p.status, 508));
      if (!ok) break;
    }
    {
      // 32 lanes x HH sums -> lane h holds head h: halve the heads while folding the lanes
      float v[HH];
#pragma unroll
      for (int h = 0; h < HH; ++h) v[h] = l_part[h];
#pragma unroll
      for (int w = HH / 2; w >= 1; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int h = 0; h < w; ++h) {
          const float give = up ? v[h] : v[h + w], keep = up ? v[h + w] : v[h];
          v[h] = keep + __shfl_xor_sync(0xffffffffu, give, w);
        }
      }
      float l = v[0];
#pragma unroll
      for (int x = HH; x < 32; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
      if (lane < HH) sums[(ob * kWorkers + warp) * 8 + lane] = make_float2(l, ref_item);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[L::bSL + ob]);
    }
    const int j_last = j0 + seg.n - 1;
    if ((j_last & (kGroups - 1)) == g) {
      ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bPV + g], (j_last / kGroups) & 1, abort_flag, p.status, 505) &&
                                       dtc_wait(&bars[L::bSL + ob], (sg / kOBufs) & 1, abort_flag, p.status, 506));
      if (!ok) break;
      tc_fence_after();
      uint32_t o[2 * HH];
      if (HH == 8) tmem_ld16(o_addr, o); else tmem_ld8(o_addr, o);
      // row sums: lane = (warp of 16, half of the heads); this warp's references are the segment's last
      float l[HH / 2];
      {
        const int w = lane & 15, h0 = (lane >> 4) * (HH / 2);
#pragma unroll
        for (int k = 0; k < HH / 2; ++k) {
          const float2 s = sums[(ob * kWorkers + w) * 8 + h0 + k];
          l[k] = s.x == 0.0f ? 0.0f : s.x * ex2_approx(s.y - ref[h0 + k]);
        }
#pragma unroll
        for (int x = 8; x >= 1; x >>= 1)
#pragma unroll
          for (int k = 0; k < HH / 2; ++k) l[k] += __shfl_xor_sync(0xffffffffu, l[k], x);
      }
      tc_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[L::bOE + ob]);
      const int e = (int)ref[8 + wq] - 127 - 8, e0 = e / 2;                       // in two factors: e can be -135
      const float back = pow2i(e0), back2 = pow2i(e - e0);
      const bool whole = seg.n == seg.n_unit;
      const size_t bh0 = (size_t)seg.b * p.H + seg.hkv * p.grp;
#pragma unroll
      for (int h = 0; h < HH; ++h) {
        const float lh = __shfl_sync(0xffffffffu, l[h % (HH / 2)], h / (HH / 2) * 16);
        if (h < p.grp) {
          const float acc = (__uint_as_float(o[h]) + __uint_as_float(o[HH + h])) * back * back2, m = ref[h];
          if (whole) {
            p.o[(bh0 + h) * 128 + kt] = __float2bfloat16_rn(acc * dtc_inverse(lh));
            if (p.lse && kt == 0) p.lse[bh0 + h] = dtc_lse(m, lh);
          } else {
            const size_t at = p.nsplit > 0 ? (bh0 + h) * p.nsplit + blockIdx.x % p.nsplit
                                           : ((size_t)blockIdx.x * 2 + (seg.t0 > 0 ? 0 : 1)) * p.grp + h;
            p.part_o[at * 128 + kt] = acc;
            if (kt == 0) { p.part_ml[at * 2] = m; p.part_ml[at * 2 + 1] = lh; }
          }
        }
      }
      __syncwarp();                                              // ref[] has been read
    }
  }
}

// One lane's four elements of query head h of a unit; heads past grp give zeros.
RK_DEVINL uint2 dtc_query_load(const DecodeTcParams& p, int b, int hkv, int h, int lane) {
  if (h >= p.grp) return make_uint2(0u, 0u);
  return __ldg(reinterpret_cast<const uint2*>(p.q + ((size_t)b * p.H + hkv * p.grp + h) * dtc::kD + lane * 4));
}
// N heads from h0 on as two MXFP8 terms each, q = hi + lo (the lib/golden block rule on q, then on the residual): a warp
// together, the heads side by side so that their shuffles overlap.
template <int HH, int N> RK_DEVINL void dtc_query_store(uint8_t* smem, const uint2 (&raw)[N], int h0, int buf, int lane) {
  using L = dtc::Lay<HH>;
  float x[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    x[i][0] = __uint_as_float(raw[i].x << 16); x[i][1] = __uint_as_float(raw[i].x & 0xFFFF0000u);
    x[i][2] = __uint_as_float(raw[i].y << 16); x[i][3] = __uint_as_float(raw[i].y & 0xFFFF0000u);
  }
#pragma unroll
  for (int term = 0; term < 2; ++term) {
    float amax[N];
#pragma unroll
    for (int i = 0; i < N; ++i) amax[i] = fmaxf(fmaxf(fabsf(x[i][0]), fabsf(x[i][1])), fmaxf(fabsf(x[i][2]), fabsf(x[i][3])));
#pragma unroll
    for (int s = 1; s < 8; s <<= 1)                                   // the 8 lanes of one 32-wide block of d
#pragma unroll
      for (int i = 0; i < N; ++i) amax[i] = fmaxf(amax[i], __shfl_xor_sync(0xffffffffu, amax[i], s));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      uint32_t code = 127u;
      float p2 = 1.0f;
      if (amax[i] > 0.0f && amax[i] < 3.0e38f) block_scale<0>(amax[i], code, p2);
      const float back = e8m0_to_f32(code);
      const uint32_t c01 = cvt_e4m3x2(x[i][1] * p2, x[i][0] * p2), c23 = cvt_e4m3x2(x[i][3] * p2, x[i][2] * p2);
      float d0, d1, d2, d3;
      e4m3x2_to_f32(c01, d1, d0);
      e4m3x2_to_f32(c23, d3, d2);
      x[i][0] -= d0 * back; x[i][1] -= d1 * back; x[i][2] -= d2 * back; x[i][3] -= d3 * back;      // residual, exact
      const int n = term * HH + h0 + i;
      *reinterpret_cast<uint32_t*>(smem + L::q_off + buf * 2048 + sw128(n, lane * 4)) = c01 | (c23 << 16);
      if ((lane & 7) == 0) smem[L::sfq_off + buf * 512 + n * 16 + (lane >> 3)] = (uint8_t)code;
    }
  }
}

template <int HH>
__global__ void __launch_bounds__(dtc::kThreads, 1)
decode_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                 const DecodeTcParams p, const uint32_t idesc_qk, const uint32_t idesc_pv) {
  using namespace dtc;
  using L = Lay<HH>;
  constexpr int kStages = L::kStages;
  extern __shared__ __align__(1024) uint8_t dtc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dtc_smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bar_off);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::misc_off + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // ---- set-up that touches nothing an earlier kernel of the stream may still be writing ------------------------------
  if (warp == kWarpQk) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  if (warp == kWarpTma && lane == 0) {
    prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
    *abort_flag = 0;
    for (int i = 0; i < kStages; ++i) mbar_init(&bars[L::bFull + i], 1);
    fence_barrier_init();
  }
  if (warp == kWarpPv) {
    for (int i = L::bEmpty + lane; i < L::nBars; i += 32) {
      const bool per_warp = i >= L::bSE && i < L::bPV;                // SE, PF, MX: the four warps of a group
      const bool four = per_warp || (i >= L::bOE && i < L::bDrain), all = i >= L::bSL && i < L::bOE;
      mbar_init(&bars[i], all ? kWorkers : four ? 4 : 1);
    }
    fence_barrier_init();
  }
  if (warp < kWorkers) {
    for (int i = threadIdx.x; i < 2 * 2048 / 16; i += kWorkers * 32) reinterpret_cast<uint4*>(smem + L::q_off)[i] = make_uint4(0u, 0u, 0u, 0u);
    // scale atoms of P, of the query terms and of V start as ones
    for (int i = threadIdx.x; i < (kGroups + 3) * 512 / 16; i += kWorkers * 32)
      reinterpret_cast<uint4*>(smem + L::sfp_off)[i] = make_uint4(0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
    // items of the exchange that no head has stay zero
    for (int i = threadIdx.x; i < kGroups * 2 * 4 * 16 / 4; i += kWorkers * 32) reinterpret_cast<uint4*>(smem + L::xchg_off)[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  grid_dependency_wait();
  grid_dependents_launch();
  const int stopped = threadIdx.x == 0 ? *reinterpret_cast<volatile int*>(p.status) : 0;
  DtcSegments seg;
  seg.start(p, lane);
  if (warp < kWorkers) fence_proxy_async_smem();                      // the fills above
  tc_fence_before();
  if (__syncthreads_or(stopped)) {                                    // an earlier launch gave up on a wait
    if (warp == kWarpQk) tmem_dealloc(*tmem_slot, kTmemCols);
    return;
  }

  auto issue_tile = [&](int j, int tile) {                            // loads of the j-th tile of this CTA
    const int st = j % kStages;
    uint8_t* sb = smem + L::stage_off + st * kStageBytes;
    const int key0 = tile * kTile, bhkv = seg.b * p.H_kv + seg.hkv;
    // scale rows past L are not read: the copy is clipped to the cache extent (L % 4 == 0 keeps it a 16-byte multiple)
    const uint32_t sbytes = (uint32_t)min(kTile, p.L - key0) * 4u;
    mbar_arrive_expect_tx(&bars[L::bFull + st], 2u * kTileBytes + 2u * sbytes);
    tma_load_3d(sb, &tmap_k, &bars[L::bFull + st], 0, key0, bhkv);
    bulk_load_1d(sb + 2 * kTileBytes, p.k_scale + ((size_t)bhkv * p.L + key0) * 4, sbytes, &bars[L::bFull + st]);
    tma_load_3d(sb + kTileBytes, &tmap_v, &bars[L::bFull + st], 0, key0, bhkv);
    bulk_load_1d(sb + 2 * kTileBytes + 512, p.v_scale + ((size_t)bhkv * p.L + key0) * 4, sbytes, &bars[L::bFull + st]);
  };
  const int n_early = min(kStages, seg.left > 0 ? seg.n : 0);         // tiles whose loads run under the rest of the set-up
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp == kWarpTma) {
    if (lane == 0)
      for (int j = 0; j < n_early; ++j) issue_tile(j, seg.t0 + j);
  } else if (warp < HH) {                                             // first query terms: the only thing S waits for beside its tile
    if (seg.left > 0) {
      const uint2 raw[1] = {dtc_query_load(p, seg.b, seg.hkv, warp, lane)};
      dtc_query_store<HH, 1>(smem, raw, warp, 0, lane);
    }
    fence_proxy_async_smem();
    asm volatile("bar.arrive 1, %0;" ::"n"((HH + 1) * 32) : "memory");
  }
  bool ok = true;

  if (warp == kWarpTma) {
    // ================= loads =================
    int j = 0;
    for (; seg.left > 0 && ok; seg.next(p)) {
      for (int i = 0; i < seg.n && ok; ++i, ++j) {
        if (j < n_early) continue;
        if (j >= kStages) ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bEmpty + j % kStages], (j / kStages - 1) & 1, abort_flag, p.status, 511));
        if (ok && lane == 0) issue_tile(j, seg.t0 + i);
      }
    }
  } else if (warp == kWarpSf) {
    // ================= key scales [key][4] -> scale atom: word (key % 32) * 4 + key / 32, in place =================
    int j = 0;
    for (; seg.left > 0 && ok; seg.next(p)) {
      for (int i = 0; i < seg.n && ok; ++i, ++j) {
        const int st = j % kStages;
        ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bFull + st], (j / kStages) & 1, abort_flag, p.status, 527));
        if (!ok) break;
        uint32_t* ks = reinterpret_cast<uint32_t*>(smem + L::stage_off + st * kStageBytes + 2 * kTileBytes);
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = ks[q * 32 + lane];
        __syncwarp();
        *reinterpret_cast<uint4*>(ks + lane * 4) = make_uint4(w[0], w[1], w[2], w[3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[L::bKS + st]);
      }
    }
  } else if (warp == kWarpQ) {
    // ================= query terms of every segment after the first, up to two segments ahead =================
    if (seg.left > 0) seg.next(p);
    for (int s = 1; seg.left > 0 && ok; ++s, seg.next(p)) {
      uint2 raw[HH];
#pragma unroll
      for (int h = 0; h < HH; ++h) raw[h] = dtc_query_load(p, seg.b, seg.hkv, h, lane);
      if (s >= 2) ok = __all_sync(0xffffffffu, dtc_wait(&bars[L::bQE + (s & 1)], ((s >> 1) - 1) & 1, abort_flag, p.status, 512));
      if (!ok) break;
      dtc_query_store<HH, HH>(smem, raw, 0, s & 1, lane);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[L::bQF + (s & 1)]);
    }
  } else if (warp == kWarpQk) {
    // ================= S^T = K Q^T (one lane) =================
    asm volatile("bar.sync 1, %0;" ::"n"((HH + 1) * 32) : "memory");
    if (lane == 0) {
      const uint64_t dk = make_smem_desc(smem_u32(smem + L::stage_off), 16, 1024, kLayoutSw128);
      const uint64_t dq = make_smem_desc(smem_u32(smem + L::q_off), 16, 1024, kLayoutSw128);
      const uint64_t dsfk = make_smem_desc(smem_u32(smem + L::stage_off + 2 * kTileBytes), 0, 128, kLayoutNone);
      tc_cp_32x128b_warpx4(tmem_base + cSfOne, make_smem_desc(smem_u32(smem + L::one_off), 0, 128, kLayoutNone));
      int j = 0;
      for (int s = 0; seg.left > 0 && ok; ++s, seg.next(p)) {
        if (s > 0) ok = dtc_wait(&bars[L::bQF + (s & 1)], (s & 1) ? (s >> 1) & 1 : ((s >> 1) - 1) & 1, abort_flag, p.status, 525);
        if (!ok) break;
        tc_cp_32x128b_warpx4(tmem_base + cSfQ + (s & 1) * 4, make_smem_desc(smem_u32(smem + L::sfq_off + (s & 1) * 512), 0, 128, kLayoutNone));
        const uint64_t dqs = dq + (uint32_t)((s & 1) * (2048 >> 4));
        for (int i = 0; i < seg.n && ok; ++i, ++j) {
          const int st = j % kStages, g = j & (kGroups - 1);
          // (the tile itself has landed: the scale warp waited for it; the second wait orders it for this thread)
          ok = dtc_wait(&bars[L::bKS + st], (j / kStages) & 1, abort_flag, p.status, 528) &&
               dtc_wait(&bars[L::bFull + st], (j / kStages) & 1, abort_flag, p.status, 521);
          if (ok && j >= kGroups) ok = dtc_wait(&bars[L::bSE + g], (j / kGroups - 1) & 1, abort_flag, p.status, 522);
          if (!ok) break;
          tc_fence_after();
          const uint32_t so = (uint32_t)(st * (kStageBytes >> 4));
          tc_cp_32x128b_warpx4(tmem_base + cSfK + st * 4, dsfk + so);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_mxf8f6f4_ss(tmem_base + cS + g * 16, dk + so + kk * 2, dqs + kk * 2, idesc_with_sf(idesc_qk, kk, kk),
                            tmem_base + cSfK + st * 4, tmem_base + cSfQ + (s & 1) * 4, kk > 0 ? 1u : 0u);
          tc_commit(&bars[L::bSF + g]);
          if (i == seg.n - 1) tc_commit(&bars[L::bQE + (s & 1)]);
        }
      }
    }
    if (lane == 0) {
      tc_commit(&bars[L::bDrain]);
      dtc_wait(&bars[L::bDrain], 0, abort_flag, p.status, 524);
    }
    __syncwarp();
  } else if (warp == kWarpPv) {
    // ================= O^T += V^T P (one lane) =================
    if (lane == 0) {
      // A = V tile [keys][d] and B = P tile [keys][n]: both have the keys as rows (32 rows of 128 bytes per instruction)
      const uint64_t dv = make_smem_desc(smem_u32(smem + L::stage_off + kTileBytes), kTileBytes, 1024, kLayoutSw128);
      const uint64_t dp = make_smem_desc(smem_u32(smem + L::p_off), kTileBytes, 1024, kLayoutSw128);
      const uint64_t dsfp = make_smem_desc(smem_u32(smem + L::sfp_off), 0, 128, kLayoutNone);
      int j = 0;
      for (int s = 0; seg.left > 0 && ok; ++s, seg.next(p)) {
        if (s >= kOBufs) ok = dtc_wait(&bars[L::bOE + s % kOBufs], (s / kOBufs - 1) & 1, abort_flag, p.status, 529);
        for (int i = 0; i < seg.n && ok; ++i, ++j) {
          const int st = j % kStages, g = j & (kGroups - 1);
          ok = dtc_wait(&bars[L::bPF + g], (j / kGroups) & 1, abort_flag, p.status, 523);
          if (!ok) break;
          tc_fence_after();
          tc_cp_32x128b_warpx4(tmem_base + cSfP + g * 4, dsfp + (uint32_t)(g * (512 >> 4)));
          const uint64_t dvt = dv + (uint32_t)(st * (kStageBytes >> 4));
          const uint64_t dpt = dp + (uint32_t)((g / L::kPerAtom) * (kTileBytes >> 4) + (g % L::kPerAtom) * (L::kNp >> 4));
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_mxf8f6f4_ss(tmem_base + cO + (s % kOBufs) * 64, dvt + kk * (4096 >> 4), dpt + kk * (4096 >> 4), idesc_with_sf(idesc_pv, kk, kk),
                            tmem_base + cSfOne, tmem_base + cSfP + g * 4, (i > 0 || kk > 0) ? 1u : 0u);
          tc_commit(&bars[L::bPV + g]);
          tc_commit(&bars[L::bEmpty + st]);
        }
      }
      tc_commit(&bars[L::bDrain + 1]);
      dtc_wait(&bars[L::bDrain + 1], 0, abort_flag, p.status, 526);
    }
    __syncwarp();
  } else {
    decode_tc_worker<HH>(p, smem, bars, tmem_base, abort_flag, seg, warp, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kWarpQk) { tc_fence_after(); tmem_dealloc(tmem_base, kTmemCols); }
}

}  // namespace rk
