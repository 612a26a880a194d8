// MX flash-attention prefill (head dim <= 128), one 128-row query tile per CTA at a time: for calls whose query tiles are few for the machine (chunks of
// a prompt, short prompts, small batches).  Stages as in fa_entry, kernels/flash_attention_mx_gqa/kernel.cpp:91-184.
//
//   warps 0-3    softmax of the even key tiles (counted over all query tiles of the CTA): thread = row (the one-lane-per-row form of
//                fused_softmax_requant_tpr, kernels/flash_attention_mx_gqa/flash_mx_impl.hpp:314-394), a row's 128 scores in the thread's registers
//   warps 4-7    softmax of the odd key tiles
//   warps 8-11   correction: rescale_accumulate (flash_mx_impl.hpp:508-532) on O in TMEM, the row sums, and O's way out; warp 8+q serves TMEM lane quadrant q
//   warp  12     TMA producer (one elected lane); hands out the work items
//   warp  13     issuer of the S = Q K^T MMAs + TMEM allocation
//   warp  14     issuer of the O += P V MMAs
//   warp  15     fills the fourth warpgroup (register reallocation works on whole warpgroups)
//
// What bounds a key tile of one query tile is the softmax of one thread's row, so two groups take key tiles in turn, half a tile apart: one forms
// exponentials (special-function unit) while the other copies S and takes maxima.  All that goes from tile to tile is the running maximum, which a group
// publishes as soon as it knows it.  S has a TMEM buffer per group, so that Q K^T is a tile ahead; O has one, and its chain from tile to tile -- P V,
// rescale, P V -- is what sets the pace now: 1 650 cycles a key tile (450 the four MMAs, 750 the rescale, the other 450 the way to the issuer and back: a few
// hundred instructions of warps that run alone and from cold instruction memory).  Without the rescale the softmax groups would take 1 580, and alone on
// the SM 1 320.  (The P V issued by a correction warp: 2 700, its other waits then lie in the chain.  The rescale in chunks of 64 columns: spills, 1 830.)
// Both groups on every key tile, 64 keys each, with an exchange of row maxima (rk_prefill2c.cu, the form for one query tile per CTA): 2 250.
// 32 heads x 509 queries behind 3581 keys 42.1 -> 35.6 us, 8 heads of 4096 69.5 -> 40.2 (pairs of query tiles), 16 of 2048 40.7 -> 27.8.
//
// As in rk_prefill2c.cu a CTA stays on its SM and takes one query tile after the other, and everything counts on from item to item.  An item costs about
// 3 600 cycles on top of its tiles: the mask of the diagonal tile, and O's way out, for which the next item's first P V waits only until O is in registers.
//
// At most two softmax warps per scheduler, and an instruction that goes to shared memory (a barrier that is complete, a load) takes them and every other
// warp some 300 cycles while the other one has exponentials queued: hence the look ahead at the end of a tile.
#include <type_traits>

#include "rk_prefill.cuh"

namespace rk {

namespace c1 {
constexpr int kStages = 3;
constexpr int kThreads = 512;
constexpr int kWarpCorr = 8, kWarpTma = 12, kWarpQk = 13, kWarpPv = 14;
// Registers of a softmax, correction and issuer thread: 128 * (2 * softmax + correction + issuer) = 65536.  Cycles of a pair of key tiles: 168 / 112 / 64
// 3 240, 160 / 120 / 72 3 290, 168 / 104 / 72 3 340, 176 / 88 / 72 3 370.
constexpr uint32_t kRegSoftmax = 168, kRegCorr = 112, kRegIssue = 64;
// TMEM columns: S of the even and of the odd key tiles, O, scale factors
constexpr uint32_t cS = 0 /* + (t & 1) * 128 */, cO = 256, cSfQ = 384 /* + buffer * 4 */, cSfK = 392 /* + st * 4 */,
                   cSfP = 404 /* + (t & 3) * 4 */, cSfV = 420 /* + st * 4 */;
// shared memory
constexpr int kPBufs = 4, kSumSlots = 8;
constexpr int q_off = 0;                                   // [2] Q tiles, taken in turn by the items
constexpr int k_off = q_off + 2 * kTileBytes;              // [3]
constexpr int v_off = k_off + kStages * kTileBytes;        // [3]
constexpr int p_off = v_off + kStages * kTileBytes;        // [4], t & 3
constexpr int stage_off = p_off + kPBufs * kTileBytes;     // [4 correction warps][2][32 rows][64 bytes]: O on its way out
constexpr int sfq_off = stage_off + 4 * 4096;              // [2]
constexpr int sfk_off = sfq_off + 2 * kSfAtomBytes;        // [3]
constexpr int sfv_off = sfk_off + kStages * kSfAtomBytes;  // [3]
constexpr int sfp_off = sfv_off + kStages * kSfAtomBytes;  // [4]
constexpr int bar_off = sfp_off + kPBufs * kSfAtomBytes;
// barrier indices (t: key tiles of the CTA, counted over all its items)
constexpr int bQ = 0 /* + Q buffer */, bKF = 2 /* + st */, bVF = 5 /* + st */, bKE = 8, bVE = 11, bSF = 14 /* + (t & 1) */, bSE = 16 /* + (t & 1) */,
              bPF = 18 /* + (t & 3) */, bPV = 22 /* + (t & 3) */, bMX = 26 /* + (t & 3) * 4 + quad */, bOR = 42 /* + (t & 1) */, bQE = 44 /* + Q buffer */,
              bDRAIN = 46, bDRAIN2 = 47, bClc = 48, bWF = 49, bWE = 50, nBars = 52;
constexpr int misc_off = bar_off + nBars * 8;              // TMEM base, abort flag
constexpr int clc_off = misc_off + 16;                     // answer of the request for the next work item
constexpr int work_off = clc_off + 16;                     // the present item, decoded (Work)
constexpr int max_off = work_off + 32;                     // [4: t & 3][128 rows] floats: running maximum of a row after key tile t
constexpr int sum_off = max_off + 4 * 128 * 4;             // [8: t & 7][128 rows] float2: sums of a row's p of key tile t, keys 0-63 and 64-127
constexpr int total = sum_off + kSumSlots * 128 * 8;
// test hook: which role sleeps a little at every key tile (schedule perturbation); kPerturbOut: at every chunk of O on its way out
constexpr int kPerturbSoftmax = 1 /* 2 = the other group */, kPerturbCorr = 3, kPerturbTma = 4, kPerturbQk = 5, kPerturbPv = 6, kPerturbOut = 7;
// One work item: a query tile of a (batch, head).
struct __align__(16) Work {
  int qt;                  // query tile; -1: no item is left
  int bh, bhkv;            // b * H + h, b * H_kv + h / group
  int n_tiles, j0;         // key tiles, first key tile inside the window
  int pad[3];
};
static_assert(sizeof(Work) == 32, "its place in shared memory");
constexpr int kReaders = 8 + 4 + 2;      // warps that read an item: softmax, correction, Q K^T, P V
}  // namespace c1

// ---- softmax warps: thread = query row, which has all 128 scores of a key tile ---------------------------------------------
// -inf into the masked scores of a key tile in TMEM (k0: its first key), by the warp of their rows.
RK_DEVINL void mask_scores_tmem(uint32_t s_addr, const PrefillParams& p, int q_pos, int k0) {
  int hi = p.S_kv - 1 - k0;                                 // masked iff c > hi || c <= lo
  if (p.causal) hi = min(hi, q_pos - k0);
  int lo = (p.window > 0) ? (q_pos - p.window - k0) : -1;
#pragma unroll 1
  for (int g = 0; g < 4; ++g, s_addr += 32, hi -= 32, lo -= 32) {
    const uint32_t keep = (hi >= 31 ? 0xffffffffu : hi < 0 ? 0u : (2u << hi) - 1u) & (lo < 0 ? 0xffffffffu : lo >= 31 ? 0u : ~((2u << lo) - 1u));
    if (__all_sync(0xffffffffu, keep == 0xffffffffu)) continue;
    uint32_t r[32];
    tmem_ld32(s_addr, r);
    tc_wait_ld();
#pragma unroll
    for (int c = 0; c < 32; ++c) r[c] = (keep & (1u << c)) ? r[c] : 0xff800000u;
    tmem_st32(s_addr, r);
  }
  tc_wait_st();
}

// The same in registers.
RK_DEVINL void mask_scores_reg(float (&s)[128], const PrefillParams& p, int q_pos, int k0) {
  int hi = p.S_kv - 1 - k0;                                 // masked iff c > hi || c <= lo
  if (p.causal) hi = min(hi, q_pos - k0);
  const int lo = (p.window > 0) ? (q_pos - p.window - k0) : -1;
#pragma unroll
  for (int c = 0; c < 128; ++c) s[c] = (c > hi || c <= lo) ? __int_as_float(0xff800000) : s[c];
}
// The maxima of the four 32-key blocks, and of all: eight independent chains (two per block), advanced in turn so that no instruction waits
// for the one before it.
RK_DEVINL float block_maxima(const float (&s)[128], float (&bmax)[4]) {
  float a0[4], a1[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    a0[g] = fmax3(s[g * 32 + 0], s[g * 32 + 1], s[g * 32 + 2]);
    a1[g] = fmax3(s[g * 32 + 3], s[g * 32 + 4], s[g * 32 + 5]);
  }
#pragma unroll
  for (int c = 6; c < 30; c += 4) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      a0[g] = fmax3(a0[g], s[g * 32 + c], s[g * 32 + c + 1]);
      a1[g] = fmax3(a1[g], s[g * 32 + c + 2], s[g * 32 + c + 3]);
    }
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) bmax[g] = fmax3(a0[g], a1[g], fmaxf(s[g * 32 + 30], s[g * 32 + 31]));
  return fmaxf(fmax3(bmax[0], bmax[1], bmax[2]), bmax[3]);
}
// p = 2^(s * sc_mul - m_use); the sums of the unquantised p of keys 0-63 and of keys 64-127; and p requantized per 32-key block into row `row` of the P tile in
// shared memory (p_row: the row's 128 bytes); returns the four E8M0 block scales.
// ex2.approx.ftz never returns a subnormal, so every non-zero p has an exponent field >= 1 and one multiply by
// 2^(7-sc) puts the E4M3 code into bits [20,27) whatever the block scale code sc is (sc < 7 needs no other
// path: all its non-zero elements lie within 2^6 of the block maximum).
RK_DEVINL uint32_t exponentiate_and_requantize(float (&s)[128], const float (&bmax)[4], float sc_mul, float m_use, uint8_t* p_row, int row, float2& sums) {
  uint64_t lsA = 0ull, lsB = 0ull;                                  // two packed pairs of partial row sums of a half
  auto half_sum = [&]() -> float {
    float ls0, ls1, ls2, ls3;
    unpack2(lsA, ls0, ls1);
    unpack2(lsB, ls2, ls3);
    lsA = lsB = 0ull;
    return (ls0 + ls1) + (ls2 + ls3);
  };
  uint32_t scale_word = 0;
  uint64_t fmul2[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const float pmax = ex2_approx(fmaf(bmax[g], sc_mul, -m_use));   // p of the block's arg-max element
    int sc = (int)(__float_as_uint(pmax) >> 23);                    // E8M0 code: se = floor(log2 pmax) <= 0
    sc = min(sc, 127);
    scale_word |= (uint32_t)sc << (8 * g);
    const float f = __uint_as_float((uint32_t)(134 - sc) << 23);   // 2^(7-sc)
    fmul2[g] = pack2(f, f);
  }
  const uint64_t sc2 = pack2(sc_mul, sc_mul), nm2 = pack2(-m_use, -m_use);
  // Four elements at a time: exponentials of block g+1 (special-function unit) next to the requantization of block
  // g (integer and FMA pipes), in one instruction stream, so that the units work side by side.
  auto exp4 = [&](int g, int c) {
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      float x0, x1;
      unpack2(fma2p(pack2(s[g * 32 + c + e], s[g * 32 + c + e + 1]), sc2, nm2), x0, x1);
      s[g * 32 + c + e] = ex2_approx(x0);
      s[g * 32 + c + e + 1] = ex2_approx(x1);
    }
  };
  // y = p * 2^(7-sc): exponent field = E4M3 exponent field, mantissa kept, so the truncated code is
  // y's bits [20,27); .ftz zeroes everything below 2^-6 of the block scale.  (The codes of four elements by two byte permutes of upper halves, two shifts
  // and a bit select, 1.25 instructions an element instead of 1.5: 2 690 cycles a pair of tiles instead of 2 560, the integer pipe is the tighter one.)
  auto requant4 = [&](int g, int c) -> uint32_t {
    const uint64_t p01 = pack2(s[g * 32 + c + 0], s[g * 32 + c + 1]);
    const uint64_t p23 = pack2(s[g * 32 + c + 2], s[g * 32 + c + 3]);
    lsA = add2p(lsA, p01);
    lsB = add2p(lsB, p23);
    uint32_t y0, y1, y2, y3;
    unpack2u(mul2p_ftz(p01, fmul2[g]), y0, y1);
    unpack2u(mul2p_ftz(p23, fmul2[g]), y2, y3);
    return pack_u8x2(y1 >> 20, y0 >> 20, pack_u8x2(y3 >> 20, y2 >> 20, 0u));
  };
#pragma unroll
  for (int c = 0; c < 32; c += 4) exp4(0, c);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (g < 3) exp4(g + 1, q * 4);
      w[q] = requant4(g, q * 4);
    }
    const int c0 = (2 * g) ^ (row & 7), c1 = (2 * g + 1) ^ (row & 7);     // 128-byte swizzle
    *reinterpret_cast<uint4*>(p_row + c0 * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(p_row + c1 * 16) = make_uint4(w[4], w[5], w[6], w[7]);
    if (g == 1) sums.x = half_sum();
  }
  sums.y = half_sum();
  return scale_word;
}

// The tiles of one item that fall to this group; t0: the CTA's key tiles of earlier items.
template <bool SOFTCAP, bool DUMP>
__device__ __forceinline__ bool softmax_every_other_tile(const PrefillParams& p, uint8_t* smem, uint64_t* bars, uint32_t tmem_base,
                                                         volatile int* abort_flag, int grp, int qt, int bh, int n_tiles, int j0, int t0) {
  using namespace c1;
  constexpr bool kMaskInTmem = !SOFTCAP;
  // With the soft cap a tile is well under way before it needs the maximum, and to wait for it at the top would put caps and maxima of the two groups in a
  // row: it is waited for where it is used.
  constexpr bool kMaxAhead = !SOFTCAP;
  uint64_t* s_full = bars + bSF + grp;
  uint64_t* s_empty = bars + bSE + grp;
  float* row_max = reinterpret_cast<float*>(smem + max_off);
  float2* row_sum = reinterpret_cast<float2*>(smem + sum_off);

  const int lane = threadIdx.x & 31;
  const int quad = (threadIdx.x >> 5) & 3;
  const int row = quad * 32 + lane;
  const uint32_t s_addr = tmem_base + (((uint32_t)(quad * 32)) << 16) + cS + grp * 128;
  const int q_pos = p.q_pos0 + qt * kBlockM + row;
  const float NEG_INF = __int_as_float(0xff800000);
  const bool dump = DUMP && p.dbg && qt == p.n_q_tiles - 1 && bh == 0;
  const float sc_mul = SOFTCAP ? 1.0f : p.scale_log2;

  bool ok = true;
  // What a tile starts with: its S, the P buffer it will write (free once the P V of four tiles before has finished) and the running maximum of the tile
  // before it, which the other group has published half a tile ago.  All three are asked for, without blocking, at the end of the group's tile before:
  // an instruction that goes to shared memory waits behind the exponentials the scheduler's other softmax warp has queued, some 300 cycles, and here
  // those of the three pass under the hand-over of P.
  bool ready = false;
  float m_run = NEG_INF;
  int fail = 0;               // which wait gave up (reported after the loops: the tile body carries no reporting code)

  // Tiles n_low .. n_high-1 need no mask for any row of this query tile: all 128 keys inside S_kv, the tile's last key not
  // beyond the first row's position, its first key inside the last row's window.
  int n_low = 0, n_high = min(n_tiles, p.S_kv / kBlockN - j0);
  {
    const int q_first = p.q_pos0 + qt * kBlockM, q_last = q_first + kBlockM - 1;
    if (p.causal) {
      const int t = q_first - (kBlockN - 1);                            // (j + j0) * kBlockN <= t
      n_high = min(n_high, t < 0 ? 0 : t / kBlockN + 1 - j0);
    }
    if (p.window > 0 && q_last >= p.window) n_low = (q_last - p.window) / kBlockN + 1 - j0;   // (j + j0) * kBlockN <= q_last - window
  }

  // the blocking forms; they return 0, or the code of the wait that gave up
  auto wait_scores = [&](const int t) -> int { return __all_sync(0xffffffffu, mbar_wait_compact(s_full, (t >> 1) & 1, abort_flag)) ? 0 : 101; };
  auto wait_rest = [&](const int j) -> int {
    const int t = t0 + j;
    int code = 0;
    if (t >= kPBufs && !mbar_wait_compact(&bars[bPV + (t & 3)], ((t >> 2) - 1) & 1, abort_flag)) code = 102;
    else if (kMaxAhead && j > 0) {
      if (!mbar_wait_compact(&bars[bMX + ((t - 1) & 3) * 4 + quad], ((t - 1) >> 2) & 1, abort_flag)) code = 106;
    }
    return __any_sync(0xffffffffu, code != 0) ? (code ? code : 102) : 0;
  };
  auto tile = [&](const int j) -> bool {
    const int t = t0 + j, pb = t & 3;                         // barriers, P buffers and slots count on from item to item; t & 1 == grp
    perturb<DUMP>(p, kPerturbSoftmax + grp, j);
    if (stops<DUMP>(p, kPerturbSoftmax + grp, j)) { fail = 101; return false; }
    const bool stamp = (quad == 0 && lane == 0);
    if (stamp) RK_STAMP(grp, j, 0);
    if (__builtin_expect(!__all_sync(0xffffffffu, ready), 0)) {       // a test issued during the group's previous tile said "not yet"
      fail = wait_scores(t);
      if (!fail) fail = wait_rest(j);
      if (fail) return false;
    }
    // Here, behind the vote on the answers, and not beside the test at the end of the tile before: a load that does not depend on the answer can be served before the test is, and
    // bring the maximum of four tiles ago beside a yes.
    if (kMaxAhead && j > 0) m_run = ld_shared_f32(&row_max[((t - 1) & 3) * 128 + row]);
    tc_fence_after();
    if (stamp) RK_STAMP(grp, j, 1);

    float s[128];
#pragma unroll
    for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + c * 32, reinterpret_cast<uint32_t*>(s) + c * 32);
    tc_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(s_empty);       // hand the S columns back: the Q K^T of the tile after the next may use them
    if (stamp) RK_STAMP(grp, j, 2);

    if (DUMP && dump && j == 0) {
#pragma unroll
      for (int c = 0; c < 128; ++c) p.dbg[row * 128 + c] = s[c];
    }

    // ---- (soft-cap,) mask, block maxima ----------------------------------------------------------------
    if (SOFTCAP) softcap_scores(s, p.scale_log2, p.cap_log2, p.inv_cap_scale);   // cap * tanh(s * scale / cap), pre-multiplied by log2 e
    if (!kMaskInTmem && __builtin_expect(j < n_low || j >= n_high, 0)) mask_scores_reg(s, p, q_pos, (j + j0) * kBlockN);
    float bmax[4];
    const float mx = block_maxima(s, bmax);
    // The running maximum follows every tile (rescale_accumulate, flash_mx_impl.hpp:508-532): it comes from the other group, which had the tile
    // before and published it half a tile ago.  (Letting it lag while the maximum grows little would save most O rescales, but p would then differ from the
    // reference's by a factor that is no power of two, its truncated E4M3 codes with it, and O by the size of the truncation noise.)
    // Barrier and slot are those of t - 5 as well: that phase is over, since the P buffer of this tile was free only after the P V of tile t - 4, for which the
    // correction warps had waited for it.
    if (!kMaxAhead && j > 0) {
      if (!__all_sync(0xffffffffu, mbar_wait_compact(&bars[bMX + ((t - 1) & 3) * 4 + quad], ((t - 1) >> 2) & 1, abort_flag))) { fail = 106; return false; }
      m_run = ld_shared_f32(&row_max[((t - 1) & 3) * 128 + row]);
    }
    const float m_new = fmaxf(m_run, mx * sc_mul);
    // Slot t & 3: a group starts tile t + 4 only when the P V of tile t is done, that is after the correction warps have read the slot, and the other
    // group has read it before its tile t + 1.
    row_max[pb * 128 + row] = m_new;
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[bMX + pb * 4 + quad]);
    // exponent = fma(s, scale, -m): lowering m by 2^-21 |m| keeps the row-max p in [1, 1 + 1e-5) in spite of
    // the rounding residue of s*scale; the common factor cancels in O = sum(p v) / sum(p).
    const float m_use = (m_new == NEG_INF) ? 0.0f : (SOFTCAP ? m_new : fmaf(-fabsf(m_new), 4.76837158203125e-7f, m_new));
    if (stamp) RK_STAMP(grp, j, 3);

    float2 sums;
    const uint32_t scale_word = exponentiate_and_requantize(s, bmax, sc_mul, m_use, smem + p_off + pb * kTileBytes + row * 128, row, sums);
    // The correction warps add them to the row's sum once this tile's P V is done.  Eight slots: the one of tile t is written again by tile t + 8, whose
    // P buffer is free when the P V of tile t + 4 is done, long after theirs of tile t + 1, at which they read it.
    row_sum[(t & (kSumSlots - 1)) * 128 + row] = sums;
    // the row's four block scales: bytes (row%32)*16 + (row/32)*4 + 0..3 of the 512-byte scale atom
    *reinterpret_cast<uint32_t*>(smem + sfp_off + pb * kSfAtomBytes + (row & 31) * 16 + (row >> 5) * 4) = scale_word;

    if (DUMP && dump && j == 0) {
      uint32_t* d32 = reinterpret_cast<uint32_t*>(p.dbg + 128 * 128);
#pragma unroll
      for (int lc = 0; lc < 8; ++lc) {
        const uint4 v4 = *reinterpret_cast<const uint4*>(smem + p_off + pb * kTileBytes + row * 128 + ((lc ^ (row & 7)) * 16));
        d32[row * 32 + lc * 4 + 0] = v4.x; d32[row * 32 + lc * 4 + 1] = v4.y;
        d32[row * 32 + lc * 4 + 2] = v4.z; d32[row * 32 + lc * 4 + 3] = v4.w;
      }
      d32[128 * 32 + row] = scale_word;
    }
    ready = j + 2 < n_tiles;                                  // the look ahead, the P buffer before the maximum (see above)
    if (ready) {
      const bool r0 = mbar_test_wait(s_full, ((t + 2) >> 1) & 1), r1 = t + 2 < kPBufs || mbar_test_wait(&bars[bPV + ((t + 2) & 3)], (((t + 2) >> 2) - 1) & 1),
                 r2 = !kMaxAhead || mbar_test_wait(&bars[bMX + ((t + 1) & 3) * 4 + quad], ((t + 1) >> 2) & 1);
      ready = r0 && r1 && r2;
    }
    if (stamp) RK_STAMP(grp, j, 4);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[bPF + pb]);
    if (stamp) RK_STAMP(grp, j, 5);
    return true;
  };

  int j = (grp ^ t0) & 1;
  if (!kMaskInTmem) {
#pragma unroll 1
    for (; j < n_tiles && ok; j += 2) ok = tile(j);
  } else {
    while (j < n_tiles && ok) {
      int end = min(n_high, n_tiles);                // a run of tiles without a mask
      if (j < n_low || j >= n_high) {                // one tile with
        fail = wait_scores(t0 + j);
        if (!fail) {
          tc_fence_after();
          mask_scores_tmem(s_addr, p, q_pos, (j + j0) * kBlockN);
          fail = wait_rest(j);
        }
        if (fail) { ok = false; break; }
        ready = true;
        end = j + 1;
      }
#pragma unroll 1
      for (; j < end && ok; j += 2) ok = tile(j);
    }
  }
  if (!ok) give_up(abort_flag, p.status, fail);
  return ok;
}

// ---- correction warps: O <- O * corr before the tile's P.V is added, the row sums, and O's way out ---------------
// What a correction thread keeps of its row.
struct RowState {
  int t;                   // the CTA's key tiles so far
  int out_qt, out_bh;      // the item the following belong to; its O is in TMEM
  float m;                 // running maximum after the last tile
  // Row sums up to the tile before it, of keys 0-63 and of keys 64-127 of the key tiles: apart until the end, as in rk_prefill2c.cu, so that a row comes
  // out the same, bit for bit, in either kernel (a call cut into smaller ones crosses from one to the other).
  float l, l_upper;
  float corr;              // factor the last tile's sums go with: l * corr + sum
};

// O / l -> bf16 of one lane quadrant (finalize_O, flash_mx_impl.hpp:535-553), a row a thread, through shared memory and TMA (a thread's own stores would
// be one sector of a line each), 32 columns at a time.
template <bool DUMP>
RK_DEVINL float finish_row(const PrefillParams& p, const uint8_t* smem, const RowState& st) {       // 1 / row sum; the log-sum-exp goes out
  const int row = threadIdx.x & 127, q_row = st.out_qt * kBlockM + row;
  const float2 sum = reinterpret_cast<const float2*>(smem + c1::sum_off)[((st.t - 1) & (c1::kSumSlots - 1)) * 128 + row];
  const float l = fmaf(st.l, st.corr, sum.x) + fmaf(st.l_upper, st.corr, sum.y);
  if (DUMP && p.dbg && st.out_qt == p.n_q_tiles - 1 && st.out_bh == 0) {
    p.dbg[128 * 128 + 128 * 32 + 128 + row * 2 + 0] = st.m;
    p.dbg[128 * 128 + 128 * 32 + 128 + row * 2 + 1] = l;
  }
  if (p.lse && q_row < p.S_q) p.lse[(size_t)st.out_bh * p.S_q + q_row] = (l > 0.0f) ? st.m * 0.6931471805599453f + logf(l) : __int_as_float(0xff800000);
  return (l > 0.0f) ? 1.0f / l : 1.0f;
}
template <int N> RK_DEVINL void scale_to_bf16(uint32_t* w, const uint32_t (&r)[N], float f) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(r[2 * i]) * f, __uint_as_float(r[2 * i + 1]) * f);
    w[i] = *reinterpret_cast<const uint32_t*>(&b2);
  }
}
RK_DEVINL void put_chunk(uint8_t* dst, const uint32_t* w) {      // 32 rows x 64 bytes, 64-byte swizzle
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(dst + lane * 64 + ((i ^ ((lane >> 1) & 3)) * 16)) = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
}
RK_DEVINL void send_chunk(const CUtensorMap* tmap_o, uint8_t* smem, int ch, int row0, int bh, const uint32_t* w) {
  const int lane = threadIdx.x & 31;
  uint8_t* dst = smem + c1::stage_off + ((threadIdx.x >> 5) & 3) * 4096 + (ch & 1) * 2048;
  if (lane == 0) bulk_wait_read<1>();             // the copy that last left this half of the stage
  __syncwarp();
  put_chunk(dst, w);
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) { tma_store_3d(tmap_o, dst, ch * 32, row0, bh); bulk_commit(); }
}
// Between two items: take_out has read all of O from TMEM when it returns, so that the next item's first P V may overwrite it; columns 64-127 are then
// still in registers and leave in send_out, off the path from one item to the next.
template <bool DUMP>
__device__ __forceinline__ void take_out(const PrefillParams& p, const CUtensorMap* tmap_o, uint8_t* smem, uint32_t tmem_base, const RowState& st, uint32_t (&w)[32]) {
  using namespace c1;
  const int quad = (threadIdx.x >> 5) & 3;
  const float inv_l = finish_row<DUMP>(p, smem, st);
  const int row0 = st.out_qt * kBlockM + quad * 32;
  tc_fence_after();
#pragma unroll 1
  for (int h = 0; h * 64 < p.d; ++h) {               // columns 0-63, 64-127
#pragma unroll
    for (int c = 0; c < 4; ++c) {                    // (32 at a time spill)
      uint32_t r[16];
      tmem_ld16(tmem_base + (((uint32_t)(quad * 32)) << 16) + cO + h * 64 + c * 16, r);
      tc_wait_ld();
      scale_to_bf16(w + 8 * c, r, inv_l);
    }
    if (h == 0 && row0 < p.S_q) {                    // (no row of the quadrant: no copies, here and in send_out; every chunk commits one otherwise, which is
      perturb<DUMP>(p, kPerturbOut, quad);           // what the wait for a half of the stage counts on)
      send_chunk(tmap_o, smem, 0, row0, st.out_bh, w);
      send_chunk(tmap_o, smem, 1, row0, st.out_bh, w + 16);
    }
  }
  tc_fence_before();
}
template <bool DUMP>
__device__ __forceinline__ void send_out(const PrefillParams& p, const CUtensorMap* tmap_o, uint8_t* smem, const RowState& st, const uint32_t (&w)[32]) {
  const int row0 = st.out_qt * kBlockM + (int)((threadIdx.x >> 5) & 3) * 32;
  if (row0 >= p.S_q || p.d <= 64) return;
  perturb<DUMP>(p, c1::kPerturbOut, 4);
  send_chunk(tmap_o, smem, 2, row0, st.out_bh, w);
  send_chunk(tmap_o, smem, 3, row0, st.out_bh, w + 16);
}
// The last item's, after which the kernel ends: straight from the registers, in fewer steps one after the other (16 heads of 300: 9.53 us through TMA, 9.35).
template <bool DUMP>
__device__ __forceinline__ void last_out(const PrefillParams& p, uint8_t* smem, uint32_t tmem_base, const RowState& st) {
  using namespace c1;
  const int quad = (threadIdx.x >> 5) & 3, q_row = st.out_qt * kBlockM + (int)(threadIdx.x & 127);
  tc_fence_after();
  __nv_bfloat16* orow = p.o + ((size_t)st.out_bh * p.S_q + q_row) * p.d;
  const bool aligned32 = (reinterpret_cast<uintptr_t>(p.o) & 31) == 0;
  float inv_l = 0.0f;
#pragma unroll 1
  for (int c = 0; c < p.d; c += 64) {
    perturb<DUMP>(p, kPerturbOut, (c >> 6) + quad);
    uint32_t r[64];
    tmem_ld32(tmem_base + (((uint32_t)(quad * 32)) << 16) + cO + c, r);
    tmem_ld32(tmem_base + (((uint32_t)(quad * 32)) << 16) + cO + c + 32, r + 32);
    if (c == 0) inv_l = finish_row<DUMP>(p, smem, st);
    tc_wait_ld();
    if (q_row < p.S_q) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(r[16 * i + 2 * e]) * inv_l, __uint_as_float(r[16 * i + 2 * e + 1]) * inv_l);
          w[e] = *reinterpret_cast<const uint32_t*>(&b2);
        }
        store_row32(orow + c + 16 * i, w, aligned32);
      }
    }
  }
}

// The tiles of one item; returns the code of the wait that gave up, or 0.
template <bool DUMP>
__device__ __forceinline__ int correct_quadrant(const PrefillParams& p, const CUtensorMap* tmap_o, uint8_t* smem, uint64_t* bars, uint32_t tmem_base,
                                                   volatile int* abort_flag, int n_tiles, RowState& st) {
  using namespace c1;
  const int lane = threadIdx.x & 31;
  const int quad = (threadIdx.x >> 5) & 3;
  const int row = quad * 32 + lane;
  const uint32_t o_addr = tmem_base + (((uint32_t)(quad * 32)) << 16) + cO;
  const float* row_max = reinterpret_cast<const float*>(smem + max_off);
  const float2* row_sum = reinterpret_cast<const float2*>(smem + sum_off);
  const float NEG_INF = __int_as_float(0xff800000);
  const int o_chunks = p.d / 32;
  auto wait_max = [&]() { return __all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bMX + (st.t & 3) * 4 + quad], (st.t >> 2) & 1, abort_flag)); };
  // Always waited for, rescale or not: an arrival on the O-ready barrier then
  // implies that its previous phase has been consumed, which is what keeps the two-deep barrier from wrapping.
  auto wait_pv = [&]() { return __all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bPV + ((st.t - 1) & 3)], ((st.t - 1) >> 2) & 1, abort_flag)); };
  auto release = [&]() {                                       // the tile's P V may accumulate into O now
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[bOR + (st.t & 1)]);
    if (quad == 0 && lane == 0) RK_STAMP(3, 0, 3);
  };
  if (n_tiles == 0) return 0;
  {                                                            // the item's first tile: nothing to rescale, but O of the item before this one to take
    uint32_t out[32];
    perturb<DUMP>(p, kPerturbCorr, 0);
    if (!wait_max()) return 401;
    const float m_new = row_max[(st.t & 3) * 128 + row];
    if (st.t > 0) {
      if (!wait_pv()) return 402;                              // (it ran under this item's first softmax)
      take_out<DUMP>(p, tmap_o, smem, tmem_base, st, out);
    }
    release();
    if (st.t > 0) send_out<DUMP>(p, tmap_o, smem, st, out);
    st.l = st.l_upper = 0.0f;
    st.corr = 1.0f;
    st.m = m_new;
    ++st.t;
  }
#pragma unroll 1
  for (int j = 1; j < n_tiles; ++j) {
    perturb<DUMP>(p, kPerturbCorr, j);
    if (stops<DUMP>(p, kPerturbCorr, j)) return 401;
    if (!wait_max()) return 401;
    const float m_new = row_max[(st.t & 3) * 128 + row];
    const float corr = (st.m == NEG_INF) ? 1.0f : ex2_approx(st.m - m_new);
    const bool rescale = __any_sync(0xffffffffu, corr != 1.0f);
    if (!wait_pv()) return 402;
    if (rescale) {
      tc_fence_after();
#pragma unroll 1
      for (int ch = 0; ch < o_chunks; ++ch) {
        uint32_t r[32];
        tmem_ld32(o_addr + ch * 32, r);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 2) mul2_ftz_inplace(r[i], r[i + 1], corr);
        tmem_st32(o_addr + ch * 32, r);
      }
      tc_wait_st();
      tc_fence_before();
    }
    release();
    const float2 sum = row_sum[((st.t - 1) & (kSumSlots - 1)) * 128 + row];       // the P V of the tile before has ended, so its sums are there
    st.l = fmaf(st.l, st.corr, sum.x);
    st.l_upper = fmaf(st.l_upper, st.corr, sum.y);
    st.corr = corr;
    st.m = m_new;
    ++st.t;
  }
  return 0;
}

template <bool SOFTCAP, bool DUMP>
__global__ void __launch_bounds__(c1::kThreads, 1)
prefill1_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const PrefillParams p, const uint32_t idesc_qk,
                 const uint32_t idesc_pv) {
  using namespace c1;
  extern __shared__ __align__(1024) uint8_t smem_raw1[];
  uint8_t* smem = align_smem(smem_raw1);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + bar_off);
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + misc_off + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) RK_STAMP(2, 0, 6);
  auto decode = [&](uint32_t block) -> Work {
    Work w;
    const Place at = place_of_block(p, block, p.n_q_tiles);
    w.qt = at.index; w.bh = at.bh; w.bhkv = at.bhkv;
    w.n_tiles = key_tiles(p, w.qt);
    // sliding window: key tiles wholly below the window of the tile's first row are masked for every row of it
    w.j0 = 0;
    if (p.window > 0) {
      const int first_key = p.q_pos0 + w.qt * kBlockM - p.window + 1;      // lowest key the first row may see
      w.j0 = min(max(first_key, 0) / kBlockN, max(w.n_tiles - 1, 0));
      w.n_tiles -= w.j0;                                                    // tiles j0 .. j0 + n_tiles - 1 are visited
    }
    w.pad[0] = w.pad[1] = w.pad[2] = 0;
    return w;
  };
  Work w = {};

  // The TMA warp sets up the barriers and goes on to its loads without waiting for the others, so that their latency runs under the
  // rest of the set-up.  Arrival counts: S-empty, P-full and O-ready take one arrival per warp of four.
  if (warp == kWarpTma) {
    for (int i = lane; i < nBars; i += 32) {
      const bool per_warp = (i >= bSE && i < bSE + 2) || (i >= bPF && i < bPF + kPBufs) || (i >= bOR && i < bOR + 2);
      mbar_init(&bars[i], per_warp ? 4 : i == bWE ? kReaders : 1);
    }
    if (lane == 0) *abort_flag = 0;
    fence_barrier_init();
    __syncwarp();
  }
  if (threadIdx.x == 0) RK_STAMP_RAW(0);
  if (warp == kWarpQk) { if (lane == 0) RK_STAMP_RAW(1); tmem_alloc(tmem_ptr, kTmemCols); tmem_relinquish(); if (lane == 0) RK_STAMP_RAW(2); }
  tc_fence_before();
  if (warp == kWarpTma) asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
  else asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
  tc_fence_after();
  if (warp != kWarpTma) {                            // (the TMA producer waits where it starts its loads)
    grid_dependency_wait();
    grid_dependents_launch();
  }
  const uint32_t tmem_base = warp == kWarpTma ? 0u : *tmem_ptr;
  if (threadIdx.x == 0) RK_STAMP_RAW(3);
  if (threadIdx.x == kWarpTma * 32) RK_STAMP_RAW(4);

  // The next item, for every warp but the TMA producer's: 1 taken, 0 none left, -1 a wait gave up.
  uint32_t work_par = 0;
  auto next_work = [&]() -> int {
    if (!__all_sync(0xffffffffu, mbar_wait_compact(&bars[bWF], work_par, abort_flag))) return -1;
    work_par ^= 1;
    w = *reinterpret_cast<const Work*>(smem + work_off);
    if (w.qt < 0) return 0;
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[bWE]);
    return 1;
  };
  constexpr int kFailWork = 501;

  // (The softmax branch comes last in the code: measured 1-1.5 % faster than first.)
  if (warp >= kWarpTma) {
    reg_dec<kRegIssue>();
    int fail = 0;                                    // which wait gave up
    // before TMEM and shared memory go back: this thread's asynchronous work has finished, also where the CTA gives up
    auto drain = [&](uint64_t* bar, uint32_t parity, int code) { if (!mbar_wait_short<true>(bar, parity, nullptr) && !fail) fail = code; };
    if (threadIdx.x == kWarpQk * 32) RK_STAMP_RAW(6);
    if (warp == kWarpTma) {
      // ================= TMA producer; hands out the items =================
      if (lane == 0) {
        prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
        int stopped = 0, kst = 0, vst = 0;           // stages of the next K and the next V tile
        bool asked = false;                          // a request for the next item is on its way
        uint32_t kuse = 0, vuse = 0, qn = 0, block = blockIdx.x;     // rounds through the stages; items with key tiles
        auto load_k = [&](int j) -> bool {
          if (kuse > 0 && !mbar_wait_compact<true>(&bars[bKE + kst], (kuse - 1) & 1, abort_flag)) { fail = 201; return false; }
          mbar_arrive_expect_tx(&bars[bKF + kst], p.kv_tile_tx + kSfAtomBytes);
          tma_load_3d(smem + k_off + kst * kTileBytes, &tmap_k, &bars[bKF + kst], 0, (j + w.j0) * kBlockN, w.bhkv);
          bulk_load_1d(smem + sfk_off + kst * kSfAtomBytes, p.k_sf + ((size_t)w.bhkv * p.n_kv_tiles + j + w.j0) * kSfAtomBytes,
                       kSfAtomBytes, &bars[bKF + kst]);
          if (++kst == kStages) { kst = 0; ++kuse; }
          return true;
        };
        // V of a tile is asked for after K of the next one, that of the next item too: a K tile then does not wait behind a V tile whose place the
        // P V of three tiles before still reads.
        int v_key = -1, v_bhkv = 0;                  // first key of the tile whose V is to come
        uint32_t v_atom = 0;
        auto load_v = [&]() -> bool {
          if (v_key < 0) return true;
          if (vuse > 0 && !mbar_wait_compact<true>(&bars[bVE + vst], (vuse - 1) & 1, abort_flag)) { fail = 202; return false; }
          mbar_arrive_expect_tx(&bars[bVF + vst], p.kv_tile_tx + kSfAtomBytes);
          tma_load_3d(smem + v_off + vst * kTileBytes, &tmap_v, &bars[bVF + vst], p.v_transposed ? v_key : 0, p.v_transposed ? 0 : v_key, v_bhkv);   // transposed V: [d][keys]
          bulk_load_1d(smem + sfv_off + vst * kSfAtomBytes, p.v_sf + (size_t)v_atom * kSfAtomBytes, kSfAtomBytes, &bars[bVF + vst]);
          if (++vst == kStages) { vst = 0; ++vuse; }
          v_key = -1;
          return true;
        };
        for (uint32_t k = 0;; ++k) {
          w = decode(block);
          // everybody has read the last item: this one takes its place
          if (k > 0 && !mbar_wait_compact<true>(&bars[bWE], (k - 1) & 1, abort_flag)) { fail = 502; break; }
          *reinterpret_cast<Work*>(smem + work_off) = w;
          mbar_arrive(&bars[bWF]);
          if (k == 0) {
            grid_dependency_wait();
            stopped = *reinterpret_cast<volatile int*>(p.status);       // an earlier launch gave up on a wait
          }
          if (w.n_tiles > 0) {
            const int qb = qn & 1;
            if (qn >= 2 && !mbar_wait_compact<true>(&bars[bQE + qb], ((qn >> 1) - 1) & 1, abort_flag)) { fail = 203; break; }
            ++qn;
            mbar_arrive_expect_tx(&bars[bQ + qb], p.q_tile_tx + kSfAtomBytes);
            tma_load_3d(smem + q_off + qb * kTileBytes, &tmap_q, &bars[bQ + qb], 0, w.qt * kBlockM, w.bh);
            bulk_load_1d(smem + sfq_off + qb * kSfAtomBytes, p.q_sf + ((size_t)w.bh * p.n_q_tiles + w.qt) * kSfAtomBytes, kSfAtomBytes, &bars[bQ + qb]);
          } else if (!load_v()) break;               // (nothing comes after which V could be asked for, and the P V issuer reads this item only when it has had it)
          // The next item is asked for three tiles before the end of this one's loads, so that the answer is there when they are under way, and not
          // earlier: the items that are left go to the SMs that are free first.
          const int ask = max(w.n_tiles - 3, 0);
#pragma unroll 1
          for (int j = 0; j < w.n_tiles || j == 0; ++j) {
            if (j == ask && !stopped) {
              mbar_arrive_expect_tx(&bars[bClc], 16);
              clc_request(smem + clc_off, &bars[bClc]);
              asked = true;
            }
            if (w.n_tiles == 0) break;
            perturb<DUMP>(p, kPerturbTma, j);
            if (stops<DUMP>(p, kPerturbTma, j)) { fail = 201; break; }
            if (!load_k(j)) break;
            if (stopped) break;                      // O is written only where V has come
            if (!load_v()) break;
            v_key = (j + w.j0) * kBlockN; v_bhkv = w.bhkv; v_atom = (uint32_t)w.bhkv * p.n_kv_tiles + j + w.j0;
          }
          if (stopped) *abort_flag = kStopped;
          if (asked) { drain(&bars[bClc], k & 1, 503); asked = false; }        // (also where the CTA gives up)
          if (fail || stopped) break;
          if (!clc_answer(smem + clc_off, block)) {
            if (!load_v()) break;
            if (!mbar_wait_compact<true>(&bars[bWE], k & 1, abort_flag)) { fail = 502; break; }
            w.qt = -1;
            *reinterpret_cast<Work*>(smem + work_off) = w;
            mbar_arrive(&bars[bWF]);
            break;
          }
          fence_proxy_async_smem();                  // the answer has been read before the next one may overwrite it
        }
        // The last loads into each place have arrived, also those whose readers have given up (this lane alone starts phases of these barriers).
        // One wait in a loop over a bit mask of barrier indices: with a wait each for K, V and Q the kernel was 0.6 % slower, by the mere size of the code.
        uint32_t want = 0, par = 0;
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
          const uint32_t nk = kuse + (i < kst), nv = vuse + (i < vst);             // loads into this stage
          want |= (uint32_t)(nk > 0) << (bKF + i) | (uint32_t)(nv > 0) << (bVF + i);
          par |= ((nk - 1) & 1) << (bKF + i) | ((nv - 1) & 1) << (bVF + i);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t nq = (qn + 1 - i) >> 1;                                   // loads into this Q buffer
          want |= (uint32_t)(nq > 0) << (bQ + i);
          par |= ((nq - 1) & 1) << (bQ + i);
        }
#pragma unroll 1
        for (; want; want &= want - 1) {
          const int b = __ffs(want) - 1;
          drain(&bars[b], (par >> b) & 1, 301);
        }
      }
      __syncwarp();
    } else if (warp == kWarpQk) {
      // ================= issuer of S = Q K^T =================
      // The whole warp runs the loop and one elected lane issues: what an MMA takes (descriptors, addresses) then is in uniform
      // registers.  (With the loop inside one lane's branch each of an MMA's operands was moved there for every MMA.)
      const uint32_t tm = warp_uniform(tmem_base);
      const uint64_t dq = make_smem_desc(smem_u32(smem + q_off), 16, 1024, kLayoutSw128);
      const uint64_t dk = make_smem_desc(smem_u32(smem + k_off), 16, 1024, kLayoutSw128);
      const uint64_t dsfq = make_smem_desc(smem_u32(smem + sfq_off), 0, 128, kLayoutNone);
      const uint64_t dsfk = make_smem_desc(smem_u32(smem + sfk_off), 0, 128, kLayoutNone);
      RK_STAMP_RAW(7);
      int st = 0, t = 0;                       // K stage; key tiles so far
      uint32_t use_par = 0, qn = 0;            // parity of the stage's use; items with key tiles
      for (int more; (more = warp_uniform(next_work())) != 0;) {
        if (more < 0) { fail = kFailWork; break; }
        const int nt = warp_uniform(w.n_tiles);
        const int qb = qn & 1;
        if (nt > 0) {
          if (!__all_sync(0xffffffffu, mbar_wait_compact(&bars[bQ + qb], (qn >> 1) & 1, abort_flag))) { fail = 301; break; }
          if (elect_one()) tc_cp_32x128b_warpx4(tm + cSfQ + qb * 4, dsfq + (uint32_t)(qb * (kSfAtomBytes >> 4)));
          ++qn;
        }
        const uint64_t dqt = dq + (uint32_t)(qb * (kTileBytes >> 4));
#pragma unroll 1
        for (int j = 0; j < nt; ++j, ++t) {
          perturb<DUMP>(p, kPerturbQk, j);
          if (stops<DUMP>(p, kPerturbQk, j)) { fail = 302; break; }
          if (lane == 0) RK_STAMP(2, j, 0);
          if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bKF + st], use_par, abort_flag))) { fail = 302; break; }
          if (t >= 2 && !__all_sync(0xffffffffu, mbar_wait_compact(&bars[bSE + (t & 1)], ((t >> 1) - 1) & 1, abort_flag))) { fail = 305; break; }
          tc_fence_after();
          if (lane == 0) RK_STAMP(2, j, 1);
          if (elect_one()) {
            tc_cp_32x128b_warpx4(tm + cSfK + st * 4, dsfk + (uint32_t)(st * (kSfAtomBytes >> 4)));
            const uint64_t dkt = dk + (uint32_t)(st * (kTileBytes >> 4));
            // rolled on purpose: this warp shares the instruction cache with the softmax warps
#pragma unroll 1
            for (int kk = 0; kk < 4; ++kk)
              mma_mxf8f6f4_ss(tm + cS + (t & 1) * 128, dqt + kk * 2, dkt + kk * 2, idesc_with_sf(idesc_qk, kk, kk), tm + cSfQ + qb * 4, tm + cSfK + st * 4, kk > 0 ? 1u : 0u);
            tc_commit(&bars[bSF + (t & 1)]);
            tc_commit(&bars[bKE + st]);
            if (j == nt - 1) tc_commit(&bars[bQE + qb]);
          }
          if (lane == 0) RK_STAMP(2, j, 2);
          if (++st == kStages) { st = 0; use_par ^= 1; }
        }
        if (fail) break;
      }
      if (elect_one()) tc_commit(&bars[bDRAIN]);
      drain(&bars[bDRAIN], 0, 306);
      __syncwarp();
    } else if (warp == kWarpPv) {
      // ================= issuer of O += P V =================
      const uint32_t tm = warp_uniform(tmem_base);
      const uint64_t dp = make_smem_desc(smem_u32(smem + p_off), 16, 1024, kLayoutSw128);
      // V tile [keys][d] is the MN-major B operand (32 keys = 32 rows of 128 bytes); a 6-bit V is stored
      // transposed and is K-major like K
      const uint64_t dv = p.v_transposed ? make_smem_desc(smem_u32(smem + v_off), 16, 1024, kLayoutSw128)
                                         : make_smem_desc(smem_u32(smem + v_off), kTileBytes, 1024, kLayoutSw128);
      const uint32_t v_kk = p.v_transposed ? 2u : (uint32_t)(4096 >> 4);
      const uint64_t dsfv = make_smem_desc(smem_u32(smem + sfv_off), 0, 128, kLayoutNone);
      const uint64_t dsfp = make_smem_desc(smem_u32(smem + sfp_off), 0, 128, kLayoutNone);
      int st = 0, t = 0;
      uint32_t use_par = 0;
      for (int more; (more = warp_uniform(next_work())) != 0;) {
        if (more < 0) { fail = kFailWork; break; }
        const int nt = warp_uniform(w.n_tiles);
#pragma unroll 1
        for (int i = 0; i < nt; ++i, ++t) {
          perturb<DUMP>(p, kPerturbPv, i);
          if (stops<DUMP>(p, kPerturbPv, i)) { fail = 303; break; }
          const int pb = t & 3;
          if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bVF + st], use_par, abort_flag))) { fail = 303; break; }
          if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bPF + pb], (t >> 2) & 1, abort_flag))) { fail = 304; break; }      // P written
          tc_fence_after();
          if (elect_one()) {
            tc_cp_32x128b_warpx4(tm + cSfV + st * 4, dsfv + (uint32_t)(st * (kSfAtomBytes >> 4)));
            tc_cp_32x128b_warpx4(tm + cSfP + pb * 4, dsfp + (uint32_t)(pb * (kSfAtomBytes >> 4)));
          }
          const uint64_t dvt = dv + (uint32_t)(st * (kTileBytes >> 4)), dpt = dp + (uint32_t)(pb * (kTileBytes >> 4));
          if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bOR + (t & 1)], (t >> 1) & 1, abort_flag))) { fail = 307; break; }      // O rescaled for this tile, or the last item's read
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_mxf8f6f4_ss(tm + cO, dpt + kk * 2, dvt + kk * v_kk, idesc_with_sf(idesc_pv, kk, kk), tm + cSfP + pb * 4, tm + cSfV + st * 4,
                              (i > 0 || kk > 0) ? 1u : 0u);
            tc_commit(&bars[bPV + pb]);
            tc_commit(&bars[bVE + st]);
          }
          if (lane == 0) RK_STAMP(2, i, 4);
          if (++st == kStages) { st = 0; use_par ^= 1; }
        }
        if (fail) break;
      }
      if (elect_one()) tc_commit(&bars[bDRAIN2]);
      drain(&bars[bDRAIN2], 0, 308);
      __syncwarp();
    }
    if (fail) give_up(abort_flag, p.status, fail);
  } else if (warp >= kWarpCorr) {
    reg_dec<kRegCorr>();
    RowState st = {};
    int fail = 0;
    for (int more; (more = next_work()) != 0;) {
      fail = more < 0 ? kFailWork : correct_quadrant<DUMP>(p, &tmap_o, smem, bars, tmem_base, abort_flag, w.n_tiles, st);
      if (fail) break;
      if (w.n_tiles > 0) { st.out_qt = w.qt; st.out_bh = w.bh; }
    }
    if (!fail && st.t > 0) {                         // O of the last item
      if (__all_sync(0xffffffffu, mbar_wait_compact(&bars[bPV + ((st.t - 1) & 3)], ((st.t - 1) >> 2) & 1, abort_flag)))
        last_out<DUMP>(p, smem, tmem_base, st);
      else fail = 403;
    }
    if (lane == 0) bulk_wait_read<0>();
    if (fail) give_up(abort_flag, p.status, fail);
  } else {
    reg_inc<kRegSoftmax>();
    if (threadIdx.x == 0) RK_STAMP_RAW(5);
    const int grp = warp >> 2;
    int t0 = 0;                                      // key tiles of earlier items
    for (int more; (more = next_work()) != 0;) {
      if (more < 0) { give_up(abort_flag, p.status, kFailWork); break; }
      if (w.n_tiles > 0) {
        if (!softmax_every_other_tile<SOFTCAP, DUMP>(p, smem, bars, tmem_base, abort_flag, grp, w.qt, w.bh, w.n_tiles, w.j0, t0)) break;
        t0 += w.n_tiles;
      } else if (grp == 0) {
        // no visible key: O = 0 (the l <= 0 guard of finalize_O, kernels/flash_attention_mx_gemma/flash_mx_impl.hpp:554-560)
        const int q_row = w.qt * kBlockM + (int)threadIdx.x;
        if (q_row < p.S_q && *reinterpret_cast<volatile int*>(p.status) == 0) {
          __nv_bfloat16* orow = p.o + ((size_t)w.bh * p.S_q + q_row) * p.d;
#pragma unroll 1
          for (int c = 0; c < p.d; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
          if (p.lse) p.lse[(size_t)w.bh * p.S_q + q_row] = __int_as_float(0xff800000);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) RK_STAMP(2, 0, 7);
  if (warp == kWarpQk) { tc_fence_after(); tmem_dealloc(tmem_base, kTmemCols); }
}

template <bool SOFTCAP, bool DUMP>
static int launch1_cfg(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                        uint32_t idesc_qk, uint32_t idesc_pv, cudaStream_t st) {
  const int smem_bytes = c1::total + 1024;
  static_assert(c1::total + 1024 <= 232448, "shared memory of a CTA");
  const dim3 grid(p.n_q_tiles * p.H * p.B);
  auto kern = prefill1_kernel<SOFTCAP, DUMP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess) return (int)e;
  if (g_ev_before && g_ev_after) cudaEventRecord(g_ev_before, st);
  e = launch_pdl(kern, grid, dim3(c1::kThreads), smem_bytes, st, tq, tk, tv, to, p, idesc_qk, idesc_pv);
  if (g_ev_before && g_ev_after) cudaEventRecord(g_ev_after, st);
  return (int)e;
}

int launch_prefill1(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                     uint32_t idesc_qk, uint32_t idesc_pv, bool softcap, cudaStream_t st) {
  if (p.dbg || p.perturb)      // the tests' stage dump and delays live in instantiations of their own: the kernels that ship carry none of their code
    return softcap ? launch1_cfg<true, true>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st) : launch1_cfg<false, true>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st);
  return softcap ? launch1_cfg<true, false>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st) : launch1_cfg<false, false>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st);
}

}  // namespace rk
