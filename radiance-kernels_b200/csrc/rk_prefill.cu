// MX flash-attention prefill for sm_100a: TMA -> shared memory -> tcgen05
// block-scaled MMA (kind::mxf8f6f4, E8M0 scales in TMEM) -> fp32 online softmax
// in registers -> P re-quantized to E4M3 + E8M0 per 32 keys -> second
// block-scaled MMA accumulating O in TMEM.
//
// Follows the streaming tile loop of fa_entry,
// kernels/flash_attention_mx_gqa/kernel.cpp:91-184 (QK_j -> fused softmax+requant
// -> scale pack -> PV_j -> rescale/accumulate -> finalize), with the stages
// mapped onto Blackwell units:
//   mxgemm_prefetch_tile / mxgemm_compute_tile (mesh)  -> TMA + tcgen05.mma
//   fused_softmax_requant_tpr (one lane per row,
//     flash_mx_impl.hpp:314-394)                       -> two threads per row, two 32-key blocks each in registers
//   pack_scales_to_sfmem (flash_mx_impl.hpp:625-639)   -> one st.shared per thread + tcgen05.cp
//   rescale_accumulate / finalize_O (:508-553)         -> O kept in TMEM, rescaled in place
//
// A CTA works on one 128-row query tile of one (batch, head) at a time.  640 threads:
//   warps 0-7   softmax of the even key tiles (counted over all query tiles of the CTA): two threads per query row (TMEM lane
//               = row), two 32-key blocks each
//   warps 8-15  softmax of the odd key tiles
//   warp  16    TMA producer (one elected lane); hands out the query tiles
//   warp  17    issuer of the S = Q K^T MMAs, TMEM allocation
//   warp  18    issuer of the O += P V MMAs: a P V that waits for its P tile never holds back the next Q K^T
//   warp  19    fills the warpgroup (registers are moved between warpgroups with setmaxnreg)
// The two groups are half a tile apart: while one forms exponentials (special-function unit) the other caps scores, takes maxima and
// rescales O (FMA and integer pipes).  All sixteen warps in the same phase of the same tile took 3600 cycles a tile with the
// cap and 2900 without; 2 x 16/8 heads of 8192: capped 974 -> 894 us, without the cap 796 -> 726, two heads of 300 keys 14.5 -> 11.9 (full clock; with what
// came after 865 capped, and 958 call after call under the power cap).
// Keys are walked in tiles of 128 (the online-softmax step, "block_n").
//
// Roofline: tensor-core bound by FLOP count (4*S_q*S_kv*d per head, half of it
// when causal); in practice the softmax/requant ALU work per S element bounds it.
#include <cuda.h>
#include <algorithm>
#include <type_traits>
#include <cuda_bf16.h>

#include "rk_common.cuh"
#include "rk_internal.h"
#include "rk_prefill.cuh"

namespace rk {

template <int DCH, int KV_STAGES>
struct SmemLayout {
  static constexpr int q_off = 0;
  static constexpr int k_off = q_off + DCH * kTileBytes;
  static constexpr int v_off = k_off + KV_STAGES * DCH * kTileBytes;
  static constexpr int p_off = v_off + KV_STAGES * DCH * kTileBytes;
  static constexpr int sfq_off = p_off + 2 * kTileBytes;
  static constexpr int sfk_off = sfq_off + DCH * kSfAtomBytes;
  static constexpr int sfv_off = sfk_off + KV_STAGES * DCH * kSfAtomBytes;
  static constexpr int sfp_off = sfv_off + KV_STAGES * DCH * kSfAtomBytes;
  static constexpr int bar_off = sfp_off + 2 * kSfAtomBytes;
  // barriers: q_full, k_full[S], k_empty[S], v_full[S], v_empty[S], s_full[2], s_empty, p_full[2], pv_done[2], drain, drain2, q_empty,
  // answer about the next item, item published, item read by all, row_bar[4 tiles][4 quadrants], end_bar[4]
  static constexpr int n_bars = 1 + 4 * KV_STAGES + 2 + 1 + 2 + 2 + 2 + 4 + 16 + 4;
  static_assert(n_bars % 2 == 0, "what follows is 16-byte aligned");
  static constexpr int misc_off = bar_off + n_bars * 8;
  static constexpr int clc_off = misc_off + 16;
  static constexpr int work_off = clc_off + 16;
  static constexpr int xchg_off = work_off + 32;              // [4 key tiles][2 parts][128 rows] floats: row maxima of a tile
  static constexpr int end_off = xchg_off + 4 * 2 * 128 * 4;  // [2 items][even, odd key tiles of the item][2 parts][128 rows] float2: row sum and its maximum
  static constexpr int total = end_off + 2 * 2 * 2 * 128 * 8;
};

// One work item: a query tile of a (batch, head).
struct __align__(16) Item {
  int qt;                  // query tile; -1: no item is left
  int bh, bhkv;            // b * H + h, b * H_kv + h / group
  int n_tiles, j0;         // key tiles, first key tile inside the window
  int pad[3];
};
static_assert(sizeof(Item) == 32, "its place in shared memory");

// test hook: which role sleeps a little at every key tile (schedule perturbation); kPerturbOut256: the upper part's warps while they write O out and
// before they hand over their shares of the row sums
constexpr int kPerturbGroup0 = 1 /* 2 = the other group */, kPerturbUpper256 = 3 /* keys 64-127 of a tile */, kPerturbTma256 = 4, kPerturbQk256 = 5,
              kPerturbPv256 = 6, kPerturbOut256 = 7;

constexpr int kNumSoftmaxWarps = 16;
constexpr int kThreads256 = (kNumSoftmaxWarps + 4) * 32;
// 512 * 104 + 128 * 64 = 640 * 96, the registers the block is launched with.  ptxas allocates by the 96, and spills 28 bytes of a thread
// (76 bytes of reloads in the code).
constexpr uint32_t kRegSoftmax256 = 104, kRegIssue256 = 64;

// What a softmax thread keeps from item to item.
struct SoftmaxState {
  int t;                   // key tiles of earlier items
  int items;               // earlier items that had key tiles
  int out_qt, out_bh;      // the last of them, whose O is still in TMEM
};
struct SoftmaxBars { uint64_t *s_full, *s_empty, *p_full, *pv_done, *row_bar, *end_bar; };

// O / l -> bf16 (finalize_O, kernels/flash_attention_mx_gqa/flash_mx_impl.hpp:535-553) by one of the two groups: a thread has half of the
// columns of its row.  The row's sum is in four shares, one per part of the item's even and of its odd key tiles, each relative to the running
// maximum its threads saw last.  They are added in that order, not in that of the groups: which group has the even tiles depends on the items
// the CTA had before, and a row must not.
template <int DCH, int KV_STAGES, bool DUMP>
__device__ __forceinline__ bool write_out_rows(const PrefillParams& p, uint8_t* smem, const SoftmaxBars& bars, uint32_t tmem_base,
                                               volatile int* abort_flag, const SoftmaxState& st) {
  using L = SmemLayout<DCH, KV_STAGES>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, part = (warp >> 2) & 1, row = quad * 32 + lane;
  const int item = st.items - 1;
  if (part == 1) perturb<DUMP>(p, kPerturbOut256, quad);
  if (!__all_sync(0xffffffffu, mbar_wait_short(&bars.end_bar[quad], item & 1, abort_flag))) return false;
  if (part == 1) perturb<DUMP>(p, kPerturbOut256, quad);      // (its partner has read the shares and goes on)
  const float2* share = reinterpret_cast<const float2*>(smem + L::end_off) + (item & 1) * 4 * 128 + row;
  const float NEG_INF = __int_as_float(0xff800000);
  const float m = fmaxf(fmaxf(share[0].y, share[128].y), fmaxf(share[256].y, share[384].y));
  float l = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) l += share[i * 128].y == NEG_INF ? share[i * 128].x : share[i * 128].x * ex2_approx(share[i * 128].y - m);      // (0, or NaN where every score was)
  const float inv_l = (l > 0.0f) ? 1.0f / l : 1.0f;
  const int q_row = st.out_qt * kBlockM + row;
  const bool live = q_row < p.S_q;
  if (DUMP && p.dbg && st.out_qt == p.n_q_tiles - 1 && st.out_bh == 0 && part == 0) {
    p.dbg[128 * 128 + 128 * 32 + 128 + row * 2 + 0] = m;
    p.dbg[128 * 128 + 128 * 32 + 128 + row * 2 + 1] = l;
  }
  if (p.lse && live && part == 0) p.lse[(size_t)st.out_bh * p.S_q + q_row] = (l > 0.0f) ? m * 0.6931471805599453f + logf(l) : NEG_INF;
  const int ncols = p.d / 2;
  const bool aligned32 = (reinterpret_cast<uintptr_t>(p.o) & 31) == 0;
  __nv_bfloat16* orow = p.o + ((size_t)st.out_bh * p.S_q + q_row) * p.d + part * ncols;
#pragma unroll 1
  for (int c = 0; c < ncols; c += 32) {
    uint32_t r[32];
    tmem_ld32(tmem_base + (((uint32_t)(quad * 32)) << 16) + kColO + part * ncols + c, r);
    tc_wait_ld();
    if (live) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
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
  return true;
}

// ---- softmax warps -----------------------------------------------------------------------------
// Group warp >> 3 takes the key tiles of its parity.  Warp w serves TMEM lane quadrant w & 3 (rows 32q..32q+31) and keys 64 * part .. + 63 of
// the tile.  A tile's row maxima go through shared memory to the row's other thread and to the other group's two, which carry the
// running maximum on to the next tile (one bounded mbarrier per tile and quadrant); each thread has its share of the row sum.
template <int DCH, int KV_STAGES, bool SOFTCAP, bool DUMP>
__device__ __forceinline__ bool softmax_rows(const PrefillParams& p, uint8_t* smem, const SoftmaxBars& bars, uint32_t tmem_base,
                                             volatile int* abort_flag, int qt, int bh, int n_tiles, int j0, SoftmaxState& state) {
  using L = SmemLayout<DCH, KV_STAGES>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = warp >> 3, part = (warp >> 2) & 1, quad = warp & 3;
  const int row = quad * 32 + lane;
  const uint32_t lane_addr = ((uint32_t)(quad * 32)) << 16;
  const float NEG_INF = __int_as_float(0xff800000);
  const float sc_mul = SOFTCAP ? 1.0f : p.scale_log2;
  float* xchg = reinterpret_cast<float*>(smem + L::xchg_off) + row;     // + ((t & 3) * 2 + part) * 128

  float m_run = NEG_INF;   // running maximum at this thread's last tile, log2 domain (score * log2 e)
  float l_run = 0.0f;      // this thread's share of the row sum, relative to it
  bool ok = true;
  // A wait for something that is there takes some 300 cycles where the scheduler's other softmax warps have exponentials queued, and a tile had four of them
  // in a row, so what it needs is asked for ahead, without blocking, and waited for only where the answer was no: 16 heads of 4096 106.7 -> 105.2 us, of 8192
  // 379 -> 369; capped, 16 of 4096 125.4 -> 123.4.  With the cap not the maxima of the tile before, which by then have been there for a while: with them
  // 124.7, and short calls 1-3 % slower than without any look ahead (4 heads of 100 8.97 -> 9.25, 2 x 16 of 1024 31.0 -> 31.7; now 8.89, 31.1).  (O in two halves of 128 columns, each rescaled under the P V of the other: 396 and 466; the issuer, alone on its warp, then sets the pace.)
  constexpr bool kMaxAhead = !SOFTCAP;
  bool s_ready = false;
  int fail = 0;            // which wait gave up

  // Tiles n_low .. n_high-1 need no mask for any row of this query tile: all 128 keys inside S_kv, the tile's last key not beyond the first
  // row's position, its first key inside the last row's window.  The body exists twice: PLAIN for those, and with the mask code.
  int n_low = 0, n_high = min(n_tiles, p.S_kv / kBlockN - j0);
  {
    const int q_first = p.q_pos0 + qt * kBlockM, q_last = q_first + kBlockM - 1;
    if (p.causal) {
      const int t = q_first - (kBlockN - 1);                            // (j + j0) * kBlockN <= t
      n_high = min(n_high, t < 0 ? 0 : t / kBlockN + 1 - j0);
    }
    if (p.window > 0 && q_last >= p.window) n_low = (q_last - p.window) / kBlockN + 1 - j0;   // (j + j0) * kBlockN <= q_last - window
  }

  auto tile = [&](const int j, auto plain_tag) -> bool {
    constexpr bool PLAIN = decltype(plain_tag)::value;
    const int t = state.t + j;                                // barriers and buffers count on from item to item; t & 1 == grp
    perturb<DUMP>(p, kPerturbGroup0 + grp, j);
    if (part == 1) perturb<DUMP>(p, kPerturbUpper256, j);
    if (stops<DUMP>(p, kPerturbGroup0 + grp, j)) { fail = 101; return false; }
    if (!__all_sync(0xffffffffu, s_ready) && !__all_sync(0xffffffffu, mbar_wait_short(&bars.s_full[grp], (t >> 1) & 1, abort_flag))) { fail = 101; return false; }
    tc_fence_after();
    float s[64];
    tmem_ld32(tmem_base + lane_addr + kColS + part * 64, reinterpret_cast<uint32_t*>(s));
    tmem_ld32(tmem_base + lane_addr + kColS + part * 64 + 32, reinterpret_cast<uint32_t*>(s) + 32);
    // Asked for here and used further down: the maxima of the tile before (the other group has left them half a tile ago), and whether the P buffer is free.
    bool last_max = j == 0, p_free = true;
    float m_last = NEG_INF;
    if (kMaxAhead && j > 0) last_max = mbar_test_wait(&bars.row_bar[((t - 1) & 3) * 4 + quad], ((t - 1) >> 2) & 1);
    if (t >= 2) p_free = mbar_test_wait(&bars.pv_done[grp], ((t - 2) >> 1) & 1);
    tc_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bars.s_empty);                 // one arrival per warp: the next Q K^T may have S once all 8 have read
    if (kMaxAhead && j > 0)
      m_last = fmaxf(ld_shared_f32_if(last_max, &xchg[((t - 1) & 3) * 256], NEG_INF), ld_shared_f32_if(last_max, &xchg[((t - 1) & 3) * 256 + 128], NEG_INF));
    if (DUMP && p.dbg && qt == p.n_q_tiles - 1 && bh == 0 && j == 0) {
#pragma unroll
      for (int c = 0; c < 64; ++c) p.dbg[row * 128 + part * 64 + c] = s[c];
    }

    // ---- (soft-cap,) mask, block maxima ------------------------------------------------------------
    // Without a cap the max is taken on the raw scores (the scale is positive) and the scale is folded
    // into the exponent's FMA; with a cap s[] is replaced by the capped score in the log2 domain.
    if (SOFTCAP) softcap_scores(s, p.scale_log2, p.cap_log2, p.inv_cap_scale);   // cap * tanh(s * scale / cap), pre-multiplied by log2 e
    if (!PLAIN) {
      const int k0 = (j + j0) * kBlockN + part * 64, q_pos = p.q_pos0 + qt * kBlockM + row;
      int hi = p.S_kv - 1 - k0;                               // masked iff c > hi || c <= lo
      if (p.causal) hi = min(hi, q_pos - k0);
      const int lo = (p.window > 0) ? (q_pos - p.window - k0) : -1;
#pragma unroll
      for (int c = 0; c < 64; ++c) s[c] = (c > hi || c <= lo) ? NEG_INF : s[c];
    }
    float bmax[2];
    {
      float a0[2], a1[2];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        a0[g] = fmax3(s[g * 32 + 0], s[g * 32 + 1], s[g * 32 + 2]);
        a1[g] = fmax3(s[g * 32 + 3], s[g * 32 + 4], s[g * 32 + 5]);
      }
#pragma unroll
      for (int c = 6; c < 30; c += 4) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          a0[g] = fmax3(a0[g], s[g * 32 + c], s[g * 32 + c + 1]);
          a1[g] = fmax3(a1[g], s[g * 32 + c + 2], s[g * 32 + c + 3]);
        }
      }
#pragma unroll
      for (int g = 0; g < 2; ++g) bmax[g] = fmax3(a0[g], a1[g], fmaxf(s[g * 32 + 30], s[g * 32 + 31]));
    }
    float tmax = fmaxf(bmax[0], bmax[1]) * sc_mul;            // -inf * positive stays -inf
    xchg[((t & 3) * 2 + part) * 128] = tmax;
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.row_bar[(t & 3) * 4 + quad]);
    if (!__all_sync(0xffffffffu, last_max)) {
      if (!__all_sync(0xffffffffu, mbar_wait_short(&bars.row_bar[((t - 1) & 3) * 4 + quad], ((t - 1) >> 2) & 1, abort_flag))) { fail = 104; return false; }
      m_last = fmaxf(xchg[((t - 1) & 3) * 256], xchg[((t - 1) & 3) * 256 + 128]);
    }
    const float m_prev = fmaxf(m_run, m_last);                // running maximum before this tile: the other group's last tile counts too
    if (!__all_sync(0xffffffffu, mbar_wait_short(&bars.row_bar[(t & 3) * 4 + quad], (t >> 2) & 1, abort_flag))) { fail = 106; return false; }
    tmax = fmaxf(tmax, xchg[((t & 3) * 2 + (part ^ 1)) * 128]);
    const float m_new = fmaxf(m_prev, tmax);
    // The exponent is formed as fma(s, scale, -m): for the row-max element that leaves the rounding
    // residue of s*scale (up to half an ulp of m) instead of exactly 0, and a p a hair below 1 would
    // drop the block scale by a binade.  Lowering the subtracted max by 2^-21 |m| keeps that p in
    // [1, 1 + 1e-5); the common factor cancels in O = sum(p v) / sum(p).
    const float m_use = (m_new == NEG_INF) ? 0.0f : (SOFTCAP ? m_new : fmaf(-fabsf(m_new), 4.76837158203125e-7f, m_new));
    const float corr = (m_prev == NEG_INF) ? 1.0f : ex2_approx(m_prev - m_new);       // of O
    const float l_corr = (m_run == NEG_INF) ? 1.0f : ex2_approx(m_run - m_new);       // of this thread's share of the sum
    m_run = m_new;
    if (!__all_sync(0xffffffffu, p_free) && !__all_sync(0xffffffffu, mbar_wait_short(&bars.pv_done[grp], ((t - 2) >> 1) & 1, abort_flag))) { fail = 107; return false; }

    // ---- p = 2^(x - m), row sum from the unquantised p, requant per 32-key block ---------------------
    // y = p * 2^(7-sc) has exponent field E - se + 7 = the E4M3 exponent field and keeps the mantissa, so the truncated code is y's
    // bits [20,27); .ftz zeroes everything below 2^-6 of the block scale.  ex2.approx.ftz never returns a subnormal, so this holds whatever sc
    // is (a block whose maximum lies below 2^-120 needs no other path: its non-zero elements all lie within 2^6 of that maximum).
    uint8_t* p_tile = smem + L::p_off + grp * kTileBytes + row * 128;
    uint64_t lsA = 0ull, lsB = 0ull;
    bool pv_there = false;
    uint32_t scale_pair = 0;
    uint64_t fmul2[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      // block max of p = 2^(block max of x - m): exp2 is monotone, so it is the p of the arg-max element; E8M0 code = its exponent field
      // (se = floor(log2 pmax) <= 0; an all-zero block gives 0)
      const float pmax = ex2_approx(fmaf(bmax[g], sc_mul, -m_use));
      const int sc = min((int)(__float_as_uint(pmax) >> 23), 127);
      scale_pair |= (uint32_t)sc << (8 * g);
      const float f = __uint_as_float((uint32_t)(134 - sc) << 23);   // 2^(7-sc)
      fmul2[g] = pack2(f, f);
    }
    const uint64_t sc2 = pack2(sc_mul, sc_mul), nm2 = pack2(-m_use, -m_use);
    auto exp4 = [&](int g, int c) {
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        float x0, x1;
        unpack2(fma2p(pack2(s[g * 32 + c + e], s[g * 32 + c + e + 1]), sc2, nm2), x0, x1);
        s[g * 32 + c + e] = ex2_approx(x0);
        s[g * 32 + c + e + 1] = ex2_approx(x1);
      }
    };
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
    for (int g = 0; g < 2; ++g) {
      uint32_t w[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (g == 0) exp4(1, q * 4);
        w[q] = requant4(g, q * 4);
      }
      if (g == 0) pv_there = t > 0 && mbar_test_wait(&bars.pv_done[grp ^ 1], ((t - 1) >> 1) & 1);
      const int c0 = (4 * part + 2 * g) ^ (row & 7), c1 = (4 * part + 2 * g + 1) ^ (row & 7);     // 128-byte swizzle
      *reinterpret_cast<uint4*>(p_tile + c0 * 16) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(p_tile + c1 * 16) = make_uint4(w[4], w[5], w[6], w[7]);
    }
    {
      float ls0, ls1, ls2, ls3;
      unpack2(lsA, ls0, ls1);
      unpack2(lsB, ls2, ls3);
      l_run = l_run * l_corr + ((ls0 + ls1) + (ls2 + ls3));
    }
    *reinterpret_cast<uint16_t*>(smem + L::sfp_off + grp * kSfAtomBytes + (row & 31) * 16 + (row >> 5) * 4 + part * 2) = (uint16_t)scale_pair;
    if (DUMP && p.dbg && qt == p.n_q_tiles - 1 && bh == 0 && j == 0) {
      // P codes as written (un-swizzled view) and the scale bytes, after the 128x128 S dump
      uint32_t* d32 = reinterpret_cast<uint32_t*>(p.dbg + 128 * 128);
#pragma unroll
      for (int lc = part * 4; lc < part * 4 + 4; ++lc) {
        const uint4 v4 = *reinterpret_cast<const uint4*>(p_tile + ((lc ^ (row & 7)) * 16));
        d32[row * 32 + lc * 4 + 0] = v4.x; d32[row * 32 + lc * 4 + 1] = v4.y;
        d32[row * 32 + lc * 4 + 2] = v4.z; d32[row * 32 + lc * 4 + 3] = v4.w;
      }
      reinterpret_cast<uint16_t*>(d32 + 128 * 32 + row)[part] = (uint16_t)scale_pair;
    }

    // ---- rescale this thread's half of the row's O in TMEM once the other group's P V has landed ----------------------
    if (t > 0) {
      if (!__all_sync(0xffffffffu, pv_there) && !__all_sync(0xffffffffu, mbar_wait_short(&bars.pv_done[grp ^ 1], ((t - 1) >> 1) & 1, abort_flag))) { fail = 102; return false; }
      tc_fence_after();
      if (j == 0) {                                           // O of the item before this one: its last P V ran under this tile's softmax
        if (!write_out_rows<DCH, KV_STAGES, DUMP>(p, smem, bars, tmem_base, abort_flag, state)) { fail = 105; return false; }
      } else if (__any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll 1
        for (int ch = 0; ch < DCH * 2; ++ch) {
          uint32_t r[32];
          const uint32_t addr = tmem_base + lane_addr + kColO + part * (DCH * 64) + ch * 32;
          tmem_ld32(addr, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 2) mul2_ftz_inplace(r[i], r[i + 1], corr);
          tmem_st32(addr, r);
        }
        tc_wait_st();
      }
    }
    s_ready = j + 2 < n_tiles && mbar_test_wait(&bars.s_full[grp], ((t + 2) >> 1) & 1);      // used at the top of the group's next tile
    fence_proxy_async_smem();   // make the st.shared P tile + scales visible to the tensor-core (async) proxy
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.p_full[grp]);
    return true;
  };

  for (int j = grp ^ (state.t & 1); j < n_tiles && ok; j += 2) {
    if (j >= n_low && j < n_high) ok = tile(j, std::true_type{});
    else ok = tile(j, std::false_type{});
  }
  if (!ok) { give_up(abort_flag, p.status, fail); return false; }
  // The shares go over by threads that had a tile of the item, and by them alone: such a thread's last tile has waited for all that the shares' readers of
  // the item before did (a P V of this item needs their O written out), so neither the shares of two items nor two phases of a barrier
  // can meet.  One that had none, for an item of one key tile, would run ahead of its own partner; the group with the tile hands over empty shares for it.
  if (part == 1) perturb<DUMP>(p, kPerturbOut256, quad);
  const int odd = grp ^ (state.t & 1);                         // this group had the item's tiles 0, 2, .. or 1, 3, ..
  if (odd < n_tiles) {
    float2* share = reinterpret_cast<float2*>(smem + L::end_off) + ((state.items & 1) * 4 + part) * 128 + row;
    share[odd * 256] = make_float2(l_run, m_run);
    if (n_tiles == 1) share[256] = make_float2(0.0f, NEG_INF);
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&bars.end_bar[quad]);
      if (n_tiles == 1) mbar_arrive(&bars.end_bar[quad]);
    }
  }
  state.t += n_tiles;
  ++state.items;
  state.out_qt = qt; state.out_bh = bh;
  return true;
}

// ---- the kernel ---------------------------------------------------------------------------------
template <int DCH, int KV_STAGES, bool SOFTCAP, bool DUMP>
__global__ void __launch_bounds__(kThreads256, 1)
prefill_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
               const __grid_constant__ CUtensorMap tmap_v, const PrefillParams p, const uint32_t idesc_qk,
               const uint32_t idesc_pv) {
  using L = SmemLayout<DCH, KV_STAGES>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = align_smem(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bar_off);
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + L::misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::misc_off + 4);

  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = k_full + KV_STAGES;
  uint64_t* v_full = k_empty + KV_STAGES;
  uint64_t* v_empty = v_full + KV_STAGES;
  uint64_t* s_full = v_empty + KV_STAGES;      // [2]: even and odd key tiles
  uint64_t* s_empty = s_full + 2;
  uint64_t* p_full = s_empty + 1;              // [2]
  uint64_t* pv_done = p_full + 2;              // [2]
  uint64_t* drain = pv_done + 2;
  uint64_t* drain2 = drain + 1;
  uint64_t* q_empty = drain2 + 1;
  uint64_t* clc_bar = q_empty + 1;
  uint64_t* work_full = clc_bar + 1;
  uint64_t* work_empty = work_full + 1;
  uint64_t* row_bar = work_empty + 1;          // [4 tiles][4 quadrants]: row maxima written
  uint64_t* end_bar = row_bar + 16;            // [4 quadrants]: row sums of an item written

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int fail = 0;                                      // which wait of an issuer gave up
  auto decode = [&](uint32_t block) -> Item {
    Item w;
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
  Item w = {};

  // The TMA warp sets up the barriers and goes on to its loads without waiting for the others, so that their latency runs under the
  // rest of the set-up.
  if (warp == kNumSoftmaxWarps) {
    if (lane == 0) {
      *abort_flag = 0;
    }
    for (int i = lane; i < L::n_bars; i += 32) {
      uint64_t* bar = bars + i;
      const int count = bar == s_empty || bar == p_full || bar == p_full + 1 ? kNumSoftmaxWarps / 2
                        : bar >= row_bar && bar < end_bar                    ? 2
                        : bar >= end_bar && bar < end_bar + 4                ? 4
                        : bar == work_empty                                  ? kNumSoftmaxWarps + 2
                                                                             : 1;
      mbar_init(bar, count);
    }
    fence_barrier_init();
    __syncwarp();
  }
  if (warp == kNumSoftmaxWarps + 1) { tmem_alloc(tmem_ptr, kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  if (warp == kNumSoftmaxWarps) asm volatile("bar.arrive 1, %0;" ::"n"(kThreads256) : "memory");
  else asm volatile("bar.sync 1, %0;" ::"n"(kThreads256) : "memory");
  tc_fence_after();
  if (warp != kNumSoftmaxWarps) {                    // (the TMA producer waits where it starts its loads)
    grid_dependency_wait();
    grid_dependents_launch();
  }
  const uint32_t tmem_base = warp == kNumSoftmaxWarps ? 0u : *tmem_ptr;

  // The next item, for every warp but the TMA producer's: 1 taken, 0 none left, -1 a wait gave up.
  uint32_t work_par = 0;
  auto next_work = [&]() -> int {
    if (!__all_sync(0xffffffffu, mbar_wait_short(work_full, work_par, abort_flag))) return -1;
    work_par ^= 1;
    w = *reinterpret_cast<const Item*>(smem + L::work_off);
    if (w.qt < 0) return 0;
    __syncwarp();
    if (lane == 0) mbar_arrive(work_empty);
    return 1;
  };
  constexpr int kFailWork = 501;

  if (warp < kNumSoftmaxWarps) {
    reg_inc<kRegSoftmax256>();
    SoftmaxState state = {0, 0, 0, 0};
    const SoftmaxBars sb = {s_full, s_empty, p_full, pv_done, row_bar, end_bar};
    int more;
    while ((more = next_work()) != 0) {
      if (more < 0) { give_up(abort_flag, p.status, kFailWork); break; }
      if (w.n_tiles > 0) {
        if (!softmax_rows<DCH, KV_STAGES, SOFTCAP, DUMP>(p, smem, sb, tmem_base, abort_flag, w.qt, w.bh, w.n_tiles, w.j0, state)) { more = -1; break; }
      } else if (warp < 4) {
        // no visible key: O = 0 (the l <= 0 guard of finalize_O, kernels/flash_attention_mx_gemma/flash_mx_impl.hpp:554-560)
        const int q_row = w.qt * kBlockM + threadIdx.x;
        if (q_row < p.S_q && *reinterpret_cast<volatile int*>(p.status) == 0) {
          __nv_bfloat16* orow = p.o + ((size_t)w.bh * p.S_q + q_row) * p.d;
#pragma unroll 1
          for (int c = 0; c < p.d; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
          if (p.lse) p.lse[(size_t)w.bh * p.S_q + q_row] = __int_as_float(0xff800000);
        }
      }
    }
    if (more == 0 && state.t > 0 && (state.t & 1) == (warp >> 3)) {      // O of the last item
      const int last = state.t - 1;
      bool ok = __all_sync(0xffffffffu, mbar_wait_short(&pv_done[last & 1], (last >> 1) & 1, abort_flag));
      if (ok) {
        tc_fence_after();
        ok = write_out_rows<DCH, KV_STAGES, DUMP>(p, smem, sb, tmem_base, abort_flag, state);
      }
      if (!ok) give_up(abort_flag, p.status, 103);
    }
  } else if (warp == kNumSoftmaxWarps) {
    // ================= TMA producer; hands out the items =================
    reg_dec<kRegIssue256>();
    if (lane == 0) {
      prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
      int stopped = 0, st = 0, q_used = 0;
      uint32_t use = 0, k_loads = 0, q_par = 0, block = blockIdx.x;
      for (uint32_t k = 0;; ++k) {
        w = decode(block);
        // everybody has read the last item: this one takes its place
        if (k > 0 && !mbar_wait_short<true>(work_empty, (k - 1) & 1, abort_flag)) { fail = 502; break; }
        *reinterpret_cast<Item*>(smem + L::work_off) = w;
        mbar_arrive(work_full);
        if (k == 0) {
          grid_dependency_wait();
          stopped = *reinterpret_cast<volatile int*>(p.status);       // an earlier launch gave up on a wait
        }
        for (int j = 0; j < w.n_tiles; ++j) {
          perturb<DUMP>(p, kPerturbTma256, j);
          if (stops<DUMP>(p, kPerturbTma256, j)) { fail = 201; break; }
          if (j == 0) {
            if (q_used) {                            // Q K^T of the last item has finished
              if (!mbar_wait_short<true>(q_empty, q_par, abort_flag)) { fail = 203; break; }
              q_par ^= 1;
            }
            q_used = 1;
            mbar_arrive_expect_tx(q_full, DCH * (p.q_tile_tx + kSfAtomBytes));
            for (int ch = 0; ch < DCH; ++ch) {
              tma_load_3d(smem + L::q_off + ch * kTileBytes, &tmap_q, q_full, ch * 128, w.qt * kBlockM, w.bh);
              bulk_load_1d(smem + L::sfq_off + ch * kSfAtomBytes,
                           p.q_sf + (((size_t)w.bh * p.n_q_tiles + w.qt) * DCH + ch) * kSfAtomBytes, kSfAtomBytes, q_full);
            }
          }
          if (use > 0 && !mbar_wait_short<true>(&k_empty[st], (use - 1) & 1, abort_flag)) { fail = 201; break; }
          mbar_arrive_expect_tx(&k_full[st], DCH * (p.kv_tile_tx + kSfAtomBytes));
          const int key = (j + w.j0) * kBlockN;
          for (int ch = 0; ch < DCH; ++ch) {
            tma_load_3d(smem + L::k_off + (st * DCH + ch) * kTileBytes, &tmap_k, &k_full[st], ch * 128, key, w.bhkv);
            bulk_load_1d(smem + L::sfk_off + (st * DCH + ch) * kSfAtomBytes,
                         p.k_sf + (((size_t)w.bhkv * p.n_kv_tiles + j + w.j0) * DCH + ch) * kSfAtomBytes, kSfAtomBytes, &k_full[st]);
          }
          ++k_loads;
          if (stopped) break;                        // O is written only where V has come
          if (use > 0 && !mbar_wait_short<true>(&v_empty[st], (use - 1) & 1, abort_flag)) { fail = 202; break; }
          mbar_arrive_expect_tx(&v_full[st], DCH * (p.kv_tile_tx + kSfAtomBytes));
          for (int ch = 0; ch < DCH; ++ch) {         // transposed V: [d][keys]
            tma_load_3d(smem + L::v_off + (st * DCH + ch) * kTileBytes, &tmap_v, &v_full[st], p.v_transposed ? key : ch * 128,
                        p.v_transposed ? ch * 128 : key, w.bhkv);
            bulk_load_1d(smem + L::sfv_off + (st * DCH + ch) * kSfAtomBytes,
                         p.v_sf + (((size_t)w.bhkv * p.n_kv_tiles + j + w.j0) * DCH + ch) * kSfAtomBytes, kSfAtomBytes, &v_full[st]);
          }
          if (++st == KV_STAGES) { st = 0; ++use; }
        }
        if (stopped) *abort_flag = kStopped;
        if (fail || stopped) break;
        // The next item is asked for now that this one's last loads are under way, and not earlier: the items that are left go to
        // the SMs that are free first.
        mbar_arrive_expect_tx(clc_bar, 16);
        clc_request(smem + L::clc_off, clc_bar);
        if (!mbar_wait_short<true>(clc_bar, k & 1, nullptr)) { fail = 503; break; }      // (also where the CTA gives up)
        if (!clc_answer(smem + L::clc_off, block)) {
          if (!mbar_wait_short<true>(work_empty, k & 1, abort_flag)) { fail = 502; break; }
          w.qt = -1;
          *reinterpret_cast<Item*>(smem + L::work_off) = w;
          mbar_arrive(work_full);
          break;
        }
        fence_proxy_async_smem();                    // the answer has been read before the next one may overwrite it
      }
      // The last loads into each place have arrived, also those whose readers have given up (this lane alone starts phases of these barriers).
      auto drain = [&](uint64_t* bar, uint32_t parity, int code) { if (!mbar_wait_short<true>(bar, parity, nullptr) && !fail) fail = code; };
      if (q_used) drain(q_full, q_par, 301);
      const uint32_t v_loads = use * KV_STAGES + st;
#pragma unroll 1
      for (uint32_t i = 0; i < KV_STAGES; ++i) {     // load n, counted from 0, is in stage n % KV_STAGES and phase n / KV_STAGES
        if (k_loads > i) drain(&k_full[i], ((k_loads - 1 - i) / KV_STAGES) & 1, 302);
        if (v_loads > i) drain(&v_full[i], ((v_loads - 1 - i) / KV_STAGES) & 1, 303);
      }
      if (fail) give_up(abort_flag, p.status, fail);
    }
    __syncwarp();
  } else if (warp == kNumSoftmaxWarps + 3) {
    reg_dec<kRegIssue256>();
  } else if (warp == kNumSoftmaxWarps + 1) {
    reg_dec<kRegIssue256>();
    // ================= issuer of S = Q K^T =================
    // The whole warp runs the loop and one elected lane issues: what an MMA takes (descriptors, addresses) then is in uniform registers.
    // Inside one lane's branch each operand was moved there for every MMA (d <= 128: 660 cycles to issue four).
    const uint32_t tm = warp_uniform(tmem_base);
    const uint64_t dq = make_smem_desc(smem_u32(smem + L::q_off), 16, 1024, kLayoutSw128);
    const uint64_t dk = make_smem_desc(smem_u32(smem + L::k_off), 16, 1024, kLayoutSw128);
    const uint64_t dsfq = make_smem_desc(smem_u32(smem + L::sfq_off), 0, 128, kLayoutNone);
    const uint64_t dsfk = make_smem_desc(smem_u32(smem + L::sfk_off), 0, 128, kLayoutNone);
    int st = 0, t = 0;                               // t: key tiles so far
    uint32_t use_par = 0, q_par = 0;
    for (int more; !fail && (more = warp_uniform(next_work())) != 0;) {
      if (more < 0) { fail = kFailWork; break; }
      const int nt = warp_uniform(w.n_tiles);
      for (int j = 0; j < nt; ++j, ++t) {
        perturb<DUMP>(p, kPerturbQk256, j);
        if (stops<DUMP>(p, kPerturbQk256, j)) { fail = 302; break; }
        if (j == 0) {
          if (!__all_sync(0xffffffffu, mbar_wait_short(q_full, q_par, abort_flag))) { fail = 301; break; }
          q_par ^= 1;
          if (elect_one()) {
  #pragma unroll
            for (int ch = 0; ch < DCH; ++ch) tc_cp_32x128b_warpx4(tm + kColSfQ + ch * 4, dsfq + (uint32_t)(ch * (kSfAtomBytes >> 4)));
          }
        }
        if (!__all_sync(0xffffffffu, mbar_wait_short(&k_full[st], use_par, abort_flag))) { fail = 302; break; }
        if (t > 0 && !__all_sync(0xffffffffu, mbar_wait_short(s_empty, (t - 1) & 1, abort_flag))) { fail = 305; break; }
        tc_fence_after();
        if (elect_one()) {
  #pragma unroll
          for (int ch = 0; ch < DCH; ++ch)
            tc_cp_32x128b_warpx4(tm + kColSfK + st * 8 + ch * 4, dsfk + (uint32_t)((st * DCH + ch) * (kSfAtomBytes >> 4)));
  #pragma unroll
          for (int ch = 0; ch < DCH; ++ch) {
            const uint64_t dqt = dq + (uint32_t)(ch * (kTileBytes >> 4));
            const uint64_t dkt = dk + (uint32_t)((st * DCH + ch) * (kTileBytes >> 4));
  #pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_mxf8f6f4_ss(tm + kColS, dqt + kk * 2, dkt + kk * 2, idesc_with_sf(idesc_qk, kk, kk), tm + kColSfQ + ch * 4, tm + kColSfK + st * 8 + ch * 4,
                              (ch > 0 || kk > 0) ? 1u : 0u);
          }
          tc_commit(&s_full[t & 1]);
          tc_commit(&k_empty[st]);
          if (j == nt - 1) tc_commit(q_empty);
        }
        if (++st == KV_STAGES) { st = 0; use_par ^= 1; }
      }
    }
    // make sure nothing issued from this warp is still running before TMEM is released
    if (elect_one()) tc_commit(drain);
    if (!mbar_wait_short<true>(drain, 0, nullptr) && !fail) fail = 306;
    if (fail) give_up(abort_flag, p.status, fail);
    __syncwarp();
  } else {
    reg_dec<kRegIssue256>();
    // ================= issuer of O += P V =================
    const uint32_t tm = warp_uniform(tmem_base);
    const uint64_t dp = make_smem_desc(smem_u32(smem + L::p_off), 16, 1024, kLayoutSw128);
    // B = V tile, MN-major (d contiguous): 32 keys = 32 rows of 128 bytes, the second 128 columns of d a tile further on; a 6-bit V
    // is stored transposed, [d][keys], and is K-major like the K tile of QK^T.
    const uint64_t dv = p.v_transposed ? make_smem_desc(smem_u32(smem + L::v_off), 16, 1024, kLayoutSw128)
                                       : make_smem_desc(smem_u32(smem + L::v_off), kTileBytes, 1024, kLayoutSw128);
    const uint32_t v_kk = p.v_transposed ? 2u : (uint32_t)(4096 >> 4);
    const uint64_t dsfp = make_smem_desc(smem_u32(smem + L::sfp_off), 0, 128, kLayoutNone);
    const uint64_t dsfv = make_smem_desc(smem_u32(smem + L::sfv_off), 0, 128, kLayoutNone);
    int st = 0, t = 0;
    uint32_t use_par = 0;
    for (int more; !fail && (more = warp_uniform(next_work())) != 0;) {
      if (more < 0) { fail = kFailWork; break; }
      const int nt = warp_uniform(w.n_tiles);
      for (int i = 0; i < nt; ++i, ++t) {
        const int pb = t & 1;
        perturb<DUMP>(p, kPerturbPv256, i);
        if (stops<DUMP>(p, kPerturbPv256, i)) { fail = 303; break; }
        if (!__all_sync(0xffffffffu, mbar_wait_short(&v_full[st], use_par, abort_flag))) { fail = 303; break; }
        if (!__all_sync(0xffffffffu, mbar_wait_short(&p_full[pb], (t >> 1) & 1, abort_flag))) { fail = 304; break; }      // (and O of the last item has been read)
        tc_fence_after();
        const uint64_t dpt = dp + (uint32_t)(pb * (kTileBytes >> 4));
        if (elect_one()) {
          tc_cp_32x128b_warpx4(tm + kColSfP + pb * 4, dsfp + (uint32_t)(pb * (kSfAtomBytes >> 4)));
  #pragma unroll
          for (int ch = 0; ch < DCH; ++ch)
            tc_cp_32x128b_warpx4(tm + kColSfV + st * 8 + ch * 4, dsfv + (uint32_t)((st * DCH + ch) * (kSfAtomBytes >> 4)));
  #pragma unroll
          for (int ch = 0; ch < DCH; ++ch) {
            const uint64_t dvt = dv + (uint32_t)((st * DCH + ch) * (kTileBytes >> 4));
  #pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_mxf8f6f4_ss(tm + kColO + ch * 128, dpt + kk * 2, dvt + kk * v_kk, idesc_with_sf(idesc_pv, kk, kk), tm + kColSfP + pb * 4,
                              tm + kColSfV + st * 8 + ch * 4, (i > 0 || kk > 0) ? 1u : 0u);
          }
          tc_commit(&pv_done[pb]);
          tc_commit(&v_empty[st]);
        }
        if (++st == KV_STAGES) { st = 0; use_par ^= 1; }
      }
    }
    if (elect_one()) tc_commit(drain2);
    if (!mbar_wait_short<true>(drain2, 0, nullptr) && !fail) fail = 308;
    if (fail) give_up(abort_flag, p.status, fail);
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kNumSoftmaxWarps + 1) { tc_fence_after(); tmem_dealloc(tmem_base, kTmemCols); }
}

// ---- host side ------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// [BH][S][d] bytes, box = 128 bytes of d x 128 rows x 1, 128-byte swizzle, rows/cols past the edge read as 0
int make_tmap_u8_3d(CUtensorMap* m, const void* base, int64_t BH, int64_t S, int64_t d) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return RK_ERR_NO_DEVICE;
  cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)S, (cuuint64_t)BH};
  cuuint64_t strides[2] = {(cuuint64_t)d, (cuuint64_t)(S * d)};
  cuuint32_t box[3] = {128, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RK_OK : RK_ERR_BAD_SHAPE;
}

// Packed 6-bit tensor [BH][rows][cols_padded codes], cols_padded a multiple of 128; a box is 128 codes x 128 rows
// and lands in shared memory as 128 bytes per row (16 codes in 12 bytes + 4 bytes of padding, 128-byte swizzle).
// bits = 4: the same with 16 codes in 8 bytes + 8 bytes of padding (16U4_ALIGN16B).
int make_tmap_sub8_3d(CUtensorMap* m, const void* base, int64_t BH, int64_t rows, int64_t cols_padded, int bits) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return RK_ERR_NO_DEVICE;
  const cuuint64_t row_bytes = (cuuint64_t)cols_padded * bits / 8;
  cuuint64_t dims[3] = {(cuuint64_t)cols_padded, (cuuint64_t)rows, (cuuint64_t)BH};
  cuuint64_t strides[2] = {row_bytes, row_bytes * (cuuint64_t)rows};
  cuuint32_t box[3] = {128, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, bits == 4 ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B : CU_TENSOR_MAP_DATA_TYPE_16U6_ALIGN16B, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RK_OK : RK_ERR_BAD_SHAPE;
}

// O, bf16 [BH][S_q][d]; a box is 32 columns x 32 rows and leaves shared memory as 64 bytes per row (64-byte swizzle).
static int make_tmap_o(CUtensorMap* m, const void* base, int64_t BH, int64_t S, int64_t d) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return RK_ERR_NO_DEVICE;
  cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)S, (cuuint64_t)BH};
  cuuint64_t strides[2] = {(cuuint64_t)(d * 2), (cuuint64_t)(S * d * 2)};
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RK_OK : RK_ERR_BAD_SHAPE;
}

template <int DCH, int KV_STAGES, bool SOFTCAP, bool DUMP>
static int launch_cfg(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const PrefillParams& p,
                      uint32_t idesc_qk, uint32_t idesc_pv, dim3 grid, cudaStream_t st) {
  using L = SmemLayout<DCH, KV_STAGES>;
  const int smem_bytes = L::total + 1024;
  auto kern = prefill_kernel<DCH, KV_STAGES, SOFTCAP, DUMP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess) return (int)e;
  if (g_ev_before && g_ev_after) cudaEventRecord(g_ev_before, st);
  e = launch_pdl(kern, grid, dim3(kThreads256), smem_bytes, st, tq, tk, tv, p, idesc_qk, idesc_pv);
  if (g_ev_before && g_ev_after) cudaEventRecord(g_ev_after, st);
  return (int)e;
}

float* g_prefill_dbg = nullptr;   // set by rk_debug_set_prefill_dump (tests only)
int g_prefill_perturb = 0, g_prefill_form = 0;

// A window that reaches beyond the first key for every row masks nothing.  Any other is at most the last row's position, so that the kernels' position - window
// - key stays within 32 bits (a caller's "no limit", a window near 2^31, wrapped and masked keys that the row sees).
static int effective_window(const rk_prefill_args& a) { return a.window > (int64_t)a.q_pos0 + a.S_q - 1 ? 0 : a.window; }

// d <= 128: one query tile per CTA at a time with the softmax groups on alternate key tiles (rk_prefill1.cu), or pairs of query tiles (rk_prefill2c.cu,
// which has a form of its own for one query tile per CTA, both groups on every key tile).  A key tile of one query tile takes 1650 cycles in the former and
// half of 3400 in the latter, which loads K and V half as often and so loses less under the power cap.  Measured (us, one call behind another in a graph, the
// attention kernel alone on prepared operands, as many KV heads as heads where no other number is given; the pairs' kernel and this one):
//   no more query tiles than SMs (both groups on every key tile, and this one): 8 / 32 heads of 512 9.0 8.3 / 9.5 9.2, 16 of 1024 14.0 12.8, 8 of 2048 23.4
//     19.9, 32 x 509 queries behind 3581 keys 37.7 32.1.  Up to three key tiles the time is that of code run for the first time, of which the other form has
//     less: 42 heads of 300 7.7 8.1, 128 of 100 6.1 6.5; over 250 calls 1.00-1.12 of its time with one key tile, 0.88-1.05 with two and three, 0.79-0.96 with more.
//     With a cap of 50 1-5 % faster, but with one of 30, where the 64 keys of a half differ in tanh's form,
//     8 of 2048 42.7 67.1, the chunk 72.0 129.
//   items of about the same length (no mask, or a long prefix): whole rounds of the SMs count.  Time of this kernel over the pairs' by rounds of the one over
//     rounds of the other, 500 calls of up to 20 rounds and 300 to 6000 keys, d of 64 and 128: without a cap 4 / 3 0.77, 3 / 2 0.78-0.95; from nine key tiles on
//     7 / 4 0.90-0.95, 11 / 6 0.95-0.99 (call after call under the power cap 0.94-1.02), 13 / 7 0.97-0.99 (1.01), 15 / 8 0.98 (1.015), 2 0.99-1.11; of six to
//     eight 7 / 4 0.98, 16 / 9 1.04-1.05; of up to five 3 / 2 0.95, 8 / 5 1.02, 7 / 4 1.01-1.02, 2 1.02-1.15 (an item costs 3600 cycles on top of its tiles here).
//     With a cap of 50 and of 30 a key tile of one query tile is 0.57-0.6 of one of a pair: 3 / 2 0.79-1.0 and 0.84-0.98 (of up to five key tiles to 1.02 and 1.17),
//     8 / 5 0.92 and 0.90, 18 / 11 1.03 and 0.95, 5 / 3 0.95-1.05 and 0.98-1.13, 7 / 4 1.01-1.11 and 0.85-1.28, 15 / 8 1.13 and 1.04.
//   others (causal, a window): short items fill the rounds up, and there are twice as many of them.  11 heads of 2048 35.7 20.3, 16 36.1 22.9, 23 36.4 31.3,
//     27 36.5 35.4; 24 heads of 1024 21.2 13.6, 37 21.5 16.9, 47 21.7 21.0; 144 of 300 16.3 14.9; 24 of 2048 with a window of 512 27.8 22.0; capped at 50 and at
//     30, 24 heads of 1024 26.6 18.6 and 64.6 33.5, 27 of 2048 53.4 51.0 and 156 134.  (Above three tiles per SM, 31 of 2048 and 56 of 1024, 2-3 % slower.)
int prefill_form(const rk_prefill_args& a, int64_t sms) {
  if (a.d > 128) return kFormWide;
  const int64_t heads = (int64_t)a.B * a.H, q_tiles = (a.S_q + kBlockM - 1) / kBlockM, tiles = q_tiles * heads, pairs = (q_tiles + 1) / 2 * heads;
  const int64_t kv_tiles = (a.S_kv + kBlockN - 1) / kBlockN;
  const int window = effective_window(a);
  const int64_t item_tiles = window > 0 ? std::min(kv_tiles, ((int64_t)window + kBlockM - 2) / kBlockN + 2) : kv_tiles;     // at most
  const bool cap = a.softcap > 0.0f;
  if (tiles <= sms) return item_tiles > 3 && !cap ? kFormTurns : kFormSplit;
  const bool level = window == 0 && (!a.causal || 2 * ((int64_t)a.q_pos0 + kBlockM) > a.S_kv);
  if (level) {
    const int64_t single_rounds = (tiles + sms - 1) / sms, pair_rounds = (pairs + sms - 1) / sms;
    const int limit = cap ? (kv_tiles <= 5 ? 149 : 160) : kv_tiles <= 5 ? 159 : kv_tiles <= 8 ? 176 : 184;       // hundredths
    return 100 * single_rounds <= limit * pair_rounds ? kFormTurns : kFormPairs;
  }
  return tiles <= 3 * sms ? kFormTurns : kFormPairs;
}

// Calls whose attention kernel prepares its operands itself (rk_prefill2c.cu, PREP): 8-bit operands with row-major scales, one query tile per CTA with both
// softmax groups on every key tile, and of those at most as many as there are stages.  Time over that of the same call with the preparation launch, 180 calls of 1 to 144 heads: one key
// tile 0.59-0.84, two 0.67-0.72 (d = 64) and 0.89-0.99 (d = 128), three 0.70-0.80 and, with six units of V for three groups of warps, 0.82-1.04: from 16 KV heads on 0.82-0.96, below 0.98-1.04.  V scaled along the keys: 0.62-0.90.
bool prefill_prepares(const rk_prefill_args& a) {
  const int kv_tiles = (a.S_kv + kBlockN - 1) / kBlockN;
  const bool rebase = a.v_scale_axis == RK_V_SCALES_ALONG_D;
  return a.d <= 128 && a.q_fmt <= RK_FMT_E5M2 && a.kv_fmt <= RK_FMT_E5M2 && a.v_scale_layout == RK_SCALES_ROWMAJOR && a.q_scale_layout == RK_SCALES_ROWMAJOR &&
         a.k_scale_layout == RK_SCALES_ROWMAJOR && a.softcap <= 0.0f && (kv_tiles < 3 || (kv_tiles == 3 && (!rebase || a.d <= 64 || (int64_t)a.B * a.H_kv >= 16))) &&
         (g_prefill_form ? g_prefill_form : prefill_form(a, num_sms())) == kFormSplit;
}

int launch_prefill(const rk_prefill_args& a, const uint8_t* q_codes, const uint8_t* k_codes, const uint8_t* v_codes,
                   const uint8_t* q_sf, const uint8_t* k_sf, const uint8_t* v_sf, bool prepares, cudaStream_t st) {
  CUtensorMap tq, tk, tv;
  int rc;
  const bool q6 = a.q_fmt >= RK_FMT_E2M3, kv6 = a.kv_fmt >= RK_FMT_E2M3;                  // packed sub-byte operands
  const int qbits = a.q_fmt == RK_FMT_E2M1 ? 4 : 6, kvbits = a.kv_fmt == RK_FMT_E2M1 ? 4 : 6;
  const int64_t dp = (a.d + 127) / 128 * 128, skp = ((int64_t)a.S_kv + 127) / 128 * 128;
  rc = q6 ? make_tmap_sub8_3d(&tq, q_codes, (int64_t)a.B * a.H, a.S_q, dp, qbits) : make_tmap_u8_3d(&tq, q_codes, (int64_t)a.B * a.H, a.S_q, a.d);
  if (rc != RK_OK) return rc;
  rc = kv6 ? make_tmap_sub8_3d(&tk, k_codes, (int64_t)a.B * a.H_kv, a.S_kv, dp, kvbits) : make_tmap_u8_3d(&tk, k_codes, (int64_t)a.B * a.H_kv, a.S_kv, a.d);
  if (rc != RK_OK) return rc;
  rc = kv6 ? make_tmap_sub8_3d(&tv, v_codes, (int64_t)a.B * a.H_kv, a.d, skp, kvbits) : make_tmap_u8_3d(&tv, v_codes, (int64_t)a.B * a.H_kv, a.S_kv, a.d);
  if (rc != RK_OK) return rc;

  PrefillParams p;
  p.q_sf = q_sf; p.k_sf = k_sf; p.v_sf = v_sf; p.v = v_codes;
  p.o = reinterpret_cast<__nv_bfloat16*>(a.o);
  p.lse = a.lse;
  p.status = device_status_word();
  if (!p.status) return RK_ERR_NO_DEVICE;
  p.dbg = g_prefill_dbg;
  p.B = a.B; p.H = a.H; p.H_kv = a.H_kv; p.S_q = a.S_q; p.S_kv = a.S_kv; p.d = a.d;
  p.group = a.H / a.H_kv;
  {
    // heads whose K and V (shared by the query heads of a KV head) fit in about 100 MB of L2, in equal groups
    const double per_head = 2.0 * a.S_kv * a.d * ((double)a.H_kv / a.H);
    const int n_bh = a.B * a.H;
    const int fit = (int)std::max(8.0, 100.0e6 / std::max(per_head, 1.0));
    const int ngroups = (n_bh + fit - 1) / fit;
    p.head_group = (n_bh + ngroups - 1) / ngroups;
  }
  p.n_q_tiles = (a.S_q + kBlockM - 1) / kBlockM;
  p.n_kv_tiles = (a.S_kv + kBlockN - 1) / kBlockN;
  p.q_pos0 = a.q_pos0; p.causal = a.causal; p.window = effective_window(a);
  p.v_transposed = kv6 ? 1 : 0;
  p.perturb = g_prefill_perturb;
  p.q_tile_tx = q6 ? kTileBytes * qbits / 8 : kTileBytes;
  p.kv_tile_tx = kv6 ? kTileBytes * kvbits / 8 : kTileBytes;
  const float scale = a.softmax_scale > 0.0f ? a.softmax_scale : 1.0f / sqrtf((float)a.d);
  p.scale_log2 = scale * 1.4426950408889634f;
  p.cap_log2 = a.softcap * 1.4426950408889634f;
  p.inv_cap_scale = a.softcap > 0.0f ? scale / a.softcap : 0.0f;

  const uint32_t idesc_qk = make_idesc(a.q_fmt, a.kv_fmt, false, false, 128, 128);
  const uint32_t idesc_pv = make_idesc(RK_FMT_E4M3, a.kv_fmt, false, /*B MN-major*/ !kv6, 128, 128);
  dim3 grid(p.n_q_tiles * a.H * a.B, 1, 1);
  const bool cap = a.softcap > 0.0f;
  if (a.d <= 128) {
    CUtensorMap to;
    rc = make_tmap_o(&to, a.o, (int64_t)a.B * a.H, a.S_q, a.d);
    if (rc != RK_OK) return rc;
    const int form = g_prefill_form ? g_prefill_form : prefill_form(a, num_sms());
    if (form == kFormTurns) return launch_prefill1(tq, tk, tv, to, p, idesc_qk, idesc_pv, cap, st);
    return launch_prefill2c(tq, tk, tv, to, p, idesc_qk, idesc_pv, cap, form == kFormSplit, !prepares ? -1 : a.v_scale_axis == RK_V_SCALES_ALONG_D ? a.kv_fmt : 2 /* its scales alone */, st);
  }
  if (p.dbg || p.perturb)      // the tests' stage dump and delays live in instantiations of their own: the kernels that ship carry none of their code
    return cap ? launch_cfg<2, 2, true, true>(tq, tk, tv, p, idesc_qk, idesc_pv, grid, st)
               : launch_cfg<2, 2, false, true>(tq, tk, tv, p, idesc_qk, idesc_pv, grid, st);
  return cap ? launch_cfg<2, 2, true, false>(tq, tk, tv, p, idesc_qk, idesc_pv, grid, st)
             : launch_cfg<2, 2, false, false>(tq, tk, tv, p, idesc_qk, idesc_pv, grid, st);
}

}  // namespace rk
