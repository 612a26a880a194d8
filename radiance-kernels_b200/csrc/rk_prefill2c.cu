// MX flash-attention prefill, two 128-row query tiles per CTA (head dim <= 128), one thread per query row and
// separate correction warps.
//
// Stages as in fa_entry, kernels/flash_attention_mx_gqa/kernel.cpp:91-184 (QK_j -> fused softmax + requant ->
// scale pack -> PV_j -> rescale/accumulate -> finalize); what this file decides is who does what:
//
//   warps 0-3    softmax of query tile A: thread = row (the one-lane-per-row form of fused_softmax_requant_tpr,
//   warps 4-7    softmax of query tile B   kernels/flash_attention_mx_gqa/flash_mx_impl.hpp:314-394): a row's 128
//                scores of a key tile sit in the thread's registers, so row max and row sum need no exchange
//   warps 8-11   correction: rescale_accumulate (flash_mx_impl.hpp:508-532) on the O accumulators in TMEM, off the
//                softmax warps' critical path, and O's way out; warp 8+q serves TMEM lane quadrant q of both tiles
//   warp  12     TMA producer (one elected lane); hands out the work items
//   warp  13     issuer of the S = Q K^T MMAs + TMEM allocation
//   warp  14     issuer of the O += P V MMAs: two issuers, so that a P V waiting for its P tile
//                never holds back the next Q K^T
//   warp  15     fills the fourth warpgroup (register reallocation works on whole warpgroups)
//
// Registers are moved between the warpgroups with setmaxnreg: the softmax threads hold a whole 128-score row
// (kRegSoftmax), correction, TMA and MMA threads need few.  The S accumulator (128 TMEM columns) is shared by the
// two tiles: a softmax group copies its rows to registers at once and hands the columns back, the Q K^T issuer
// alternates QK_A, QK_B.  Every K/V tile brought in by TMA serves both query tiles.
//
// A CTA stays on its SM and takes one pair of query tiles after the other: the grid has a block per pair, and a running CTA
// takes over the index of one that has not started (cluster launch control).  All barriers, buffers and slots count on from item to
// item, so nothing drains in between: the next item's loads start while the last tiles of this one are worked on, group A goes
// on while group B, one tile longer under a causal mask, finishes, and the correction warps write an item's O out while the softmax
// warps are in their next tile.  With a CTA per pair an item of 16 tiles cost 17 000 cycles on top of them (start 4400, first loads,
// a masked tile in cold code, the last tile of B alone, epilogue 3700): 8 x 16 heads of 4096 620 -> 518 us, 4 x 32 / 8 heads of
// 8192 2030 -> 1764 us at full clock; call after call under the power cap 619 -> 555 and 2036 -> 1890.  Since the waits outside the softmax
// warps are short in code (mbar_wait_compact) and the registers split as below, 534 and 1838 under the cap (544 and 1857 before them on the same machine).
//
// SPLIT: one query tile per CTA and no second item, for grids that leave SMs idle and whose items are too short for rk_prefill1.cu, or capped.  A key
// tile's time is then the softmax of one thread's row (about 3200 cycles for 128 scores, the tensor core waits), so both softmax groups work
// on the same tile, group A on keys 0-63 of each key tile and group B on keys 64-127, and exchange their row maxima through
// shared memory.
//
// SPLIT with PREP = the format of K and V (E4M3, E5M2; kPrepScales where V is scaled along the keys): the preparation of a small call, which is otherwise a launch of its own.  The issuers and the warp that fills the warpgroup put the
// row-major scales of Q and K into atoms, softmax and correction warps re-block V, scaled along d, into the stages V is read from, in the time Q and K take to arrive and the
// first scores to be formed: there is a stage for every key tile.  A query tile of every head re-blocks V for itself, so this is for items of at most three key tiles and grids
// of one round of the SMs.  (A launch whose results the next one waits for costs 1.2 us,
// its own chain of latencies 2 to 4.)  Without a mask, us a call: one head of 256 keys, d = 64, 9.2 -> 6.3; 32 / 8 heads of 128 keys, d = 128, 7.1 -> 5.8; 8 x 18 heads of 128 10.6 -> 6.9; 40
// heads of 384, d = 128, 12.6 -> 10.5, d = 64, 12.0 -> 8.7.
#include <type_traits>

#include "rk_prefill.cuh"
#include "rk_rebase.cuh"

namespace rk {

namespace c2 {
constexpr int kStages = 3;
constexpr int kThreads = 512;
constexpr int kWarpCorr = 8, kWarpTma = 12, kWarpQk = 13, kWarpPv = 14;
// Registers of a softmax, correction and issuer thread: 128 * (2 * softmax + correction + issuer) = 65536.  Measured (8 x 16 heads of
// 4096, full clock): softmax 168 515 us, 176 518, 184 521, 192 523, 200 550 (no spills up to 192; what changes is the order ptxas gives the tile body).
// With the short waits, 4 x 32 / 8 of 8192 under the power cap: 168 / 104 / 72 1858 us, 168 / 96 / 80 1860, 168 / 88 / 88 1857, 176 / 88 / 72 1866, 176 / 80 / 80 1868;
// 32 / 8 heads of 8192 445.1, 446.4, 445.2, 448.0, 448.2.  The capped form is 1 % slower with 168 (2 x 16 heads of 4096 213.6 and 216.0; 8 x 16 784 and 791).
template <bool SOFTCAP> constexpr uint32_t kRegSoftmax = SOFTCAP ? 176 : 168;
template <bool SOFTCAP> constexpr uint32_t kRegCorr = SOFTCAP ? 88 : 104;
constexpr uint32_t kRegIssue = 72;
static_assert(2 * kRegSoftmax<false> + kRegCorr<false> + kRegIssue == 512 && 2 * kRegSoftmax<true> + kRegCorr<true> + kRegIssue == 512);
constexpr uint32_t kRegSoftmaxSplit = 176, kRegCorrSplit = 80, kRegIssueSplit = 80;      // 509 queries behind 3581 keys: softmax 144 43.9 us, 160 44.4, 176 43.5, 192 43.6
// TMEM columns
constexpr uint32_t cS = 0, cO = 128 /* + g*128 */, cSfQ = 384 /* + g*4 */, cSfK = 392 /* + st*4 */,
                   cSfP = 404 /* + (g*2+pb)*4 */, cSfV = 420 /* + st*4 */;
// shared memory
constexpr int q_off = 0;                                   // [2][16 KB]
constexpr int k_off = q_off + 2 * kTileBytes;              // [3]
constexpr int v_off = k_off + kStages * kTileBytes;        // [3]
constexpr int p_off = v_off + kStages * kTileBytes;        // [2 groups][2]
constexpr int stage_off = p_off + 4 * kTileBytes;          // [4 correction warps][2][32 rows][64 bytes]: O on its way out
constexpr int sfq_off = stage_off + 4 * 4096;              // [2]
constexpr int sfk_off = sfq_off + 2 * kSfAtomBytes;        // [3]
constexpr int sfv_off = sfk_off + kStages * kSfAtomBytes;  // [3]
constexpr int sfp_off = sfv_off + kStages * kSfAtomBytes;  // [2][2]
constexpr int bar_off = sfp_off + 4 * kSfAtomBytes;
// barrier indices
constexpr int bQ = 0 /* group A's; group B's is bQB */, bKF = 1, bKE = 4, bVF = 7, bVE = 10, bSF = 13 /* +g */, bSE = 15 /* +g */,
              bPF = 17 /* + g*2+pb */, bPV = 21 /* + g*2+pb */, bCF = 25 /* + (g*4+slot)*4+quad */, bOR = 57 /* + g*2+pb */,
              bDRAIN = 61, bDRAIN2 = 62, bQE = 63 /* +g */, bClc = 65, bWF = 66, bWE = 67, bQB = 68, nBars = 70;
constexpr int misc_off = bar_off + nBars * 8;              // TMEM base, abort flag
constexpr int clc_off = misc_off + 16;                     // answer of the request for the next work item
constexpr int work_off = clc_off + 16;                     // the present item, decoded (Work)
constexpr int corr_off = work_off + 32;                    // [2 groups][4 slots][128] floats: the O rescale factors of a tile; in the slot of an
                                                           // item's first tile, which has none, 1 / row sum of the item before
constexpr int lse_off = corr_off + 2 * 4 * 128 * 4;        // the same places: log-sum-exp of the rows of the item before
constexpr int total = lse_off + 2 * 4 * 128 * 4;
// test hook: which role sleeps a little at every key tile (schedule perturbation); kPerturbOut: at every chunk of O on its way out, and between the
// softmax warps' last tile of an item and what they leave for it
// PREP: kPerturbAtoms before the scale atoms of Q and of each key tile, kPerturbV before each unit of V; where these stop, some warps do not hand over (all but Q's;
// the upper three quarters of V's keys, or its last tile's scales) and the waits for them run out.
constexpr int kPerturbSoftmaxA = 1 /* 2 = softmax of tile B (SPLIT: of keys 64-127) */, kPerturbCorr = 3, kPerturbTma = 4, kPerturbQk = 5, kPerturbPv = 6,
              kPerturbOut = 7, kPerturbAtoms = 8, kPerturbV = 9;
// One work item: a pair of query tiles (SPLIT: one) of a (batch, head).
struct __align__(16) Work {
  int qp;                  // pair index; -1: no item is left
  int bh, bhkv;            // b * H + h, b * H_kv + h / group
  int nt0, nt1;            // key tiles of its two query tiles
  int j0;                  // first key tile inside the window
  int pad[2];
};
static_assert(sizeof(Work) == 32, "its place in shared memory");
constexpr int kReaders = 8 + 4 + 2;      // warps that read an item: softmax, correction, Q K^T, P V
constexpr int bPrep = bClc;              // PREP: the scale atoms of Q and K are there (no second item is asked for)
constexpr int kPrepScales = 2;           // PREP beside the formats: V is scaled along the keys and comes as it lies, only its scales have to be put into atoms
}  // namespace c2

// ---- softmax warps: thread = query row -----------------------------------------------------------------------
// The loop over key tiles is what runs nearly all the time, and it is kept small: an SM's instruction cache holds 32 KB, a body is
// 15 KB of straight-line code, and code that is not in the cache runs at a third of the speed.  So there is one body; the few
// tiles that need a mask (the causal diagonal, the end of the keys, the edge of a window) have it written into their scores in
// TMEM beforehand by a short loop.  (With the soft cap the mask has to come after the cap, and with SPLIT a body is half as long:
// those keep a second body, PLAIN or not.)  The stage dump (tests) exists only in the DUMP instantiation of the kernel.
template <int G>
__device__ __forceinline__ void mask_scores(uint32_t s_addr, const PrefillParams& p, int q_pos, int k0) {
  int hi = p.S_kv - 1 - k0;                                 // masked iff c > hi || c <= lo
  if (p.causal) hi = min(hi, q_pos - k0);
  int lo = (p.window > 0) ? (q_pos - p.window - k0) : -1;
#pragma unroll 1
  for (int g = 0; g < G; ++g, s_addr += 32, hi -= 32, lo -= 32) {
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

// The blocking form of the two waits a key tile starts with (its S, and the P buffer it will write), for tiles whose
// early tests said "not yet".  Inline: as a function call it made the kernel 23 % slower.  Returns 0, or the code of the wait that gave up.
__device__ __forceinline__ int wait_tile_inputs(uint64_t* s_full, uint32_t s_parity, uint64_t* pv_done, uint32_t pv_parity,
                                             int need_pv, volatile int* abort_flag) {
  if (!mbar_wait_short(s_full, s_parity, abort_flag)) return 101;
  if (need_pv && !mbar_wait_short(pv_done, pv_parity, abort_flag)) return 102;
  return 0;
}

template <bool SOFTCAP, bool DUMP, bool SPLIT>
__device__ __forceinline__ bool softmax_row_group(const PrefillParams& p, uint8_t* smem, uint64_t* bars, uint32_t tmem_base,
                                                  volatile int* abort_flag, int grp, int qt, int bh, int n_tiles, int j0, int t0) {
  using namespace c2;
  const int half = SPLIT ? grp : 0;                 // which 64 keys of a tile
  if (SPLIT) grp = 0;                               // query tile of this CTA whose barriers, P and O it uses
  constexpr int kN = SPLIT ? 64 : 128, kG = kN / 32;   // this thread's scores of a key tile, their 32-key blocks
  constexpr bool kMaskInTmem = !SOFTCAP && !SPLIT;
  uint64_t* s_full = bars + bSF + grp;
  uint64_t* s_empty = bars + bSE + grp;
  uint64_t* p_full = bars + bPF + grp * 2;
  uint64_t* pv_done = bars + bPV + grp * 2;
  uint64_t* corr_full = bars + bCF + grp * 16;
  float* corr_sm = reinterpret_cast<float*>(smem + corr_off) + grp * 512;
  // SPLIT: the two groups' exchange, in the place of tile B's rescale factors: [2 tiles][2 halves][128 rows]
  uint64_t* xchg_bar = bars + bCF + 16;
  float* xchg = reinterpret_cast<float*>(smem + corr_off) + 512;

  const int lane = threadIdx.x & 31;
  const int quad = (threadIdx.x >> 5) & 3;
  const int row = quad * 32 + lane;
  const uint32_t lane_addr = ((uint32_t)(quad * 32)) << 16;
  const int q_row = qt * kBlockM + row;
  const int q_pos = p.q_pos0 + q_row;
  const float NEG_INF = __int_as_float(0xff800000);
  const bool dump = DUMP && p.dbg && qt == p.n_q_tiles - 1 && bh == 0;
  const float sc_mul = SOFTCAP ? 1.0f : p.scale_log2;

  // The row's sum is kept apart for the two halves of the key tiles, whether one thread has both or, with SPLIT, one each: a row comes
  // out the same, bit for bit, in either form (a call cut into smaller ones crosses from one form to the other).
  float m_run = NEG_INF, l_run = 0.0f, l_upper = 0.0f;
  bool ok = true;
  bool s_ready = false;       // results of early, non-blocking tests of the next tile's S barrier and P buffer
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

  auto tile = [&](const int j, auto plain_tag) -> bool {
    constexpr bool PLAIN = decltype(plain_tag)::value;
    const int t = t0 + j, pb = t & 1;                         // barriers, P buffers and rescale slots count on from item to item
    perturb<DUMP>(p, kPerturbSoftmaxA + (SPLIT ? half : grp), j);
    if (stops<DUMP>(p, kPerturbSoftmaxA + (SPLIT ? half : grp), j)) { fail = 101; return false; }
    const bool stamp = (quad == 0 && lane == 0);
    if (stamp) RK_STAMP(grp, j, 0);
    if (__builtin_expect(!__all_sync(0xffffffffu, s_ready), 0)) {   // a test issued during the previous tile said "not yet"
      const int w = wait_tile_inputs(s_full, t & 1, &pv_done[pb], ((t - 2) >> 1) & 1, t >= 2, abort_flag);
      if (__any_sync(0xffffffffu, w != 0)) { fail = w ? w : 101; return false; }
    }
    tc_fence_after();
    if (stamp) RK_STAMP(grp, j, 1);

    // first key of this tile (j counts from the first tile inside the window), and of this thread's scores
    const int key0 = (j + j0) * kBlockN, k0 = key0 + half * 64;

    float s[kN];
#pragma unroll
    for (int c = 0; c < kG; ++c) tmem_ld32(tmem_base + lane_addr + cS + half * 64 + c * 32, reinterpret_cast<uint32_t*>(s) + c * 32);
    tc_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(s_empty);       // hand the S columns back: the other query tile's QK^T may use them
    if (stamp) RK_STAMP(grp, j, 2);

    if (DUMP && dump && j == 0) {
#pragma unroll
      for (int c = 0; c < kN; ++c) p.dbg[row * 128 + half * 64 + c] = s[c];
    }

    // ---- (soft-cap,) mask, block maxima ----------------------------------------------------------------
    if (SOFTCAP) softcap_scores(s, p.scale_log2, p.cap_log2, p.inv_cap_scale);   // cap * tanh(s * scale / cap), pre-multiplied by log2 e
    if (!kMaskInTmem && !PLAIN && (j < n_low || j >= n_high)) {
      int hi = p.S_kv - 1 - k0;                               // masked iff c > hi || c <= lo
      if (p.causal) hi = min(hi, q_pos - k0);
      const int lo = (p.window > 0) ? (q_pos - p.window - k0) : -1;
#pragma unroll
      for (int c = 0; c < kN; ++c) s[c] = (c > hi || c <= lo) ? NEG_INF : s[c];
    }
    // block maxima: eight independent chains (two per 32-key block), advanced in turn so that no instruction waits
    // for the one before it
    float bmax[kG];
    {
      float a0[kG], a1[kG];
#pragma unroll
      for (int g = 0; g < kG; ++g) {
        a0[g] = fmax3(s[g * 32 + 0], s[g * 32 + 1], s[g * 32 + 2]);
        a1[g] = fmax3(s[g * 32 + 3], s[g * 32 + 4], s[g * 32 + 5]);
      }
#pragma unroll
      for (int c = 6; c < 30; c += 4) {
#pragma unroll
        for (int g = 0; g < kG; ++g) {
          a0[g] = fmax3(a0[g], s[g * 32 + c], s[g * 32 + c + 1]);
          a1[g] = fmax3(a1[g], s[g * 32 + c + 2], s[g * 32 + c + 3]);
        }
      }
#pragma unroll
      for (int g = 0; g < kG; ++g) bmax[g] = fmax3(a0[g], a1[g], fmaxf(s[g * 32 + 30], s[g * 32 + 31]));
    }
    float mx;
    if (SPLIT) {
      mx = fmaxf(bmax[0], bmax[1]);
      float* xr = xchg + (j & 1) * 256 + row;
      xr[half * 128] = mx;
      __syncwarp();
      if (lane == 0) mbar_arrive(&xchg_bar[(j & 3) * 4 + quad]);
      const bool met = mbar_wait_short(&xchg_bar[(j & 3) * 4 + quad], (j >> 2) & 1, abort_flag);
      if (!__all_sync(0xffffffffu, met)) { fail = 106; return false; }
      mx = fmaxf(mx, xr[(half ^ 1) * 128]);
    } else {
      mx = fmaxf(fmax3(bmax[0], bmax[1], bmax[kG - 2]), bmax[kG - 1]);
    }
    // The running maximum follows every tile (rescale_accumulate, flash_mx_impl.hpp:508-532).  Letting it lag
    // while the maximum grows little would save most O rescales, but p would then differ from the reference's by a
    // factor that is no power of two, its truncated E4M3 codes with it, and O by the size of the truncation noise.
    const float m_new = fmaxf(m_run, mx * sc_mul);
    // exponent = fma(s, scale, -m): lowering m by 2^-21 |m| keeps the row-max p in [1, 1 + 1e-5) in spite of
    // the rounding residue of s*scale; the common factor cancels in O = sum(p v) / sum(p).
    const float m_use = (m_new == NEG_INF) ? 0.0f : (SOFTCAP ? m_new : fmaf(-fabsf(m_new), 4.76837158203125e-7f, m_new));
    const float corr = (m_run == NEG_INF) ? 1.0f : ex2_approx(m_run - m_new);
    m_run = m_new;
    // The correction warp of this lane quadrant can start on O while the exponentials run here.  Slot t & 3: this
    // group is never more than two tiles ahead of the correction warp (the wait for the P buffer at the top of the
    // tile sees to that), so a slot is free again long before it comes round.
    if (!SPLIT || half == 0) {
      if (SPLIT || j > 0) corr_sm[(t & 3) * 128 + row] = corr;     // (j = 0: left there at the end of the last item)
      __syncwarp();
      if (lane == 0) mbar_arrive(&corr_full[(t & 3) * 4 + quad]);
    }
    if (stamp) RK_STAMP(grp, j, 3);

    // ---- p = 2^(x - m), row sum from the unquantised p, requant per 32-key block ---------------------
    // ex2.approx.ftz never returns a subnormal, so every non-zero p has an exponent field >= 1 and one multiply by
    // 2^(7-sc) puts the E4M3 code into bits [20,27) whatever the block scale code sc is (sc < 7 needs no other
    // path: all its non-zero elements lie within 2^6 of the block maximum).
    uint8_t* p_tile = smem + p_off + (grp * 2 + pb) * kTileBytes + row * 128;
    uint64_t lsA = 0ull, lsB = 0ull;                                  // two packed pairs of partial row sums of a half
    auto add_half = [&](float& l) {
      float ls0, ls1, ls2, ls3;
      unpack2(lsA, ls0, ls1);
      unpack2(lsB, ls2, ls3);
      l = fmaf(l, corr, (ls0 + ls1) + (ls2 + ls3));
      lsA = lsB = 0ull;
    };
    uint32_t scale_word = 0;
    uint64_t fmul2[kG];
#pragma unroll
    for (int g = 0; g < kG; ++g) {
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
    // y's bits [20,27); .ftz zeroes everything below 2^-6 of the block scale.
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
    for (int g = 0; g < kG; ++g) {
      uint32_t w[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (g < kG - 1) exp4(g + 1, q * 4);
        w[q] = requant4(g, q * 4);
      }
      const int c0 = (4 * half + 2 * g) ^ (row & 7), c1 = (4 * half + 2 * g + 1) ^ (row & 7);     // 128-byte swizzle
      *reinterpret_cast<uint4*>(p_tile + c0 * 16) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(p_tile + c1 * 16) = make_uint4(w[4], w[5], w[6], w[7]);
      if (g == 1) add_half(l_run);
    }
    if (!SPLIT) add_half(l_upper);
    // the row's four block scales: bytes (row%32)*16 + (row/32)*4 + 0..3 of the 512-byte scale atom
    uint8_t* sf = smem + sfp_off + (grp * 2 + pb) * kSfAtomBytes + (row & 31) * 16 + (row >> 5) * 4;
    if (SPLIT) *reinterpret_cast<uint16_t*>(sf + half * 2) = (uint16_t)scale_word;
    else *reinterpret_cast<uint32_t*>(sf) = scale_word;

    if (DUMP && dump && j == 0) {
      uint32_t* d32 = reinterpret_cast<uint32_t*>(p.dbg + 128 * 128);
#pragma unroll
      for (int lc = half * 4; lc < half * 4 + 2 * kG; ++lc) {
        const uint4 v4 = *reinterpret_cast<const uint4*>(p_tile + ((lc ^ (row & 7)) * 16));
        d32[row * 32 + lc * 4 + 0] = v4.x; d32[row * 32 + lc * 4 + 1] = v4.y;
        d32[row * 32 + lc * 4 + 2] = v4.z; d32[row * 32 + lc * 4 + 3] = v4.w;
      }
      if (SPLIT) reinterpret_cast<uint16_t*>(d32 + 128 * 32 + row)[half] = (uint16_t)scale_word;
      else d32[128 * 32 + row] = scale_word;
    }
    // a look ahead at the next tile's S barrier and at its P buffer (free once the P.V that read it two tiles
    // before has finished): asked here, used at the top of the next tile
    s_ready = (j + 1 < n_tiles) && mbar_test_wait(s_full, (t + 1) & 1) &&
              (t < 1 || mbar_test_wait(&pv_done[(t + 1) & 1], ((t - 1) >> 1) & 1));
    if (stamp) RK_STAMP(grp, j, 4);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&p_full[pb]);
    if (stamp) RK_STAMP(grp, j, 5);
    return true;
  };

  int j = 0;
  if (!kMaskInTmem) {
    if (n_low == 0)
      for (; j < n_high && ok; ++j) ok = tile(j, std::true_type{});
    for (; j < n_tiles && ok; ++j) ok = tile(j, std::false_type{});
  } else {
    while (j < n_tiles && ok) {
      int end = min(n_high, n_tiles);                // a run of tiles without a mask
      if (j < n_low || j >= n_high) {                // one tile with
        const int t = t0 + j;
        const int w = wait_tile_inputs(s_full, t & 1, &pv_done[t & 1], ((t - 2) >> 1) & 1, t >= 2, abort_flag);
        if (__any_sync(0xffffffffu, w != 0)) { fail = w ? w : 101; ok = false; break; }
        tc_fence_after();
        mask_scores<kG>(tmem_base + lane_addr + cS, p, q_pos, (j + j0) * kBlockN);
        s_ready = true;
        end = j + 1;
      }
#pragma unroll 1
      for (; j < end && ok; ++j) ok = tile(j, std::true_type{});
    }
  }
  if (SPLIT && ok) {                                                    // the row's sum: both halves
    float* xr = xchg + (n_tiles & 1) * 256 + row;
    xr[half * 128] = l_run;
    __syncwarp();
    if (lane == 0) mbar_arrive(&xchg_bar[(n_tiles & 3) * 4 + quad]);
    ok = __all_sync(0xffffffffu, mbar_wait_short(&xchg_bar[(n_tiles & 3) * 4 + quad], (n_tiles >> 2) & 1, abort_flag));
    if (!ok) fail = 107;
    if (ok) l_upper = xr[(half ^ 1) * 128];
  }
  l_run += l_upper;

  // ---- epilogue: O / l -> bf16 (finalize_O, flash_mx_impl.hpp:535-553) ----------------------------------------
  if (SPLIT && ok) {
    const int last = t0 + n_tiles - 1;
    ok = __all_sync(0xffffffffu, mbar_wait_short(&pv_done[last & 1], (last >> 1) & 1, abort_flag));
    if (!ok) fail = 103;
  }
  if (!ok) give_up(abort_flag, p.status, fail);
  if (ok) {
    const float inv_l = (l_run > 0.0f) ? 1.0f / l_run : 1.0f;
    const float lse = (l_run > 0.0f) ? m_run * 0.6931471805599453f + logf(l_run) : NEG_INF;
    const bool live = q_row < p.S_q;
    if (DUMP && dump) {
      p.dbg[128 * 128 + 128 * 32 + 128 + row * 2 + 0] = m_run;
      p.dbg[128 * 128 + 128 * 32 + 128 + row * 2 + 1] = l_run;
    }
    if (!SPLIT) {
      // The correction warps write O out when the group's next tile asks for the accumulator (the arrival on its rescale factor, or
      // the one after the last item, covers these stores); the group goes on to that tile at once.
      perturb<DUMP>(p, kPerturbOut, quad);
      const int slot = (t0 + n_tiles) & 3;
      corr_sm[slot * 128 + row] = inv_l;
      reinterpret_cast<float*>(smem + lse_off)[(grp * 4 + slot) * 128 + row] = lse;
      return true;
    }
    if (p.lse && live && half == 0) p.lse[(size_t)bh * p.S_q + q_row] = lse;
    tc_fence_after();
    if (quad == 0 && lane == 0) RK_STAMP(grp, 0, 6);
    __nv_bfloat16* orow = p.o + ((size_t)bh * p.S_q + q_row) * p.d;
    const bool aligned32 = (reinterpret_cast<uintptr_t>(p.o) & 31) == 0;
    // the row's registers are free now: this group's half of the columns is fetched with one wait
    const int c32_0 = half * (p.d / 64), n_c32 = c32_0 + p.d / 64;
#pragma unroll 1
    for (int h = c32_0; h < n_c32; h += 2) {
      uint32_t r[64];
      tmem_ld32(tmem_base + lane_addr + cO + grp * 128 + h * 32, r);
      if (h + 1 < n_c32) tmem_ld32(tmem_base + lane_addr + cO + grp * 128 + (h + 1) * 32, r + 32);
      tc_wait_ld();
      if (live) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (h + c < n_c32) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t w[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const float* f = reinterpret_cast<const float*>(r) + c * 32 + i * 16 + 2 * e;
                const __nv_bfloat162 b2 = __floats2bfloat162_rn(f[0] * inv_l, f[1] * inv_l);
                w[e] = *reinterpret_cast<const uint32_t*>(&b2);
              }
              store_row32(orow + (h + c) * 32 + i * 16, w, aligned32);
            }
          }
        }
      }
    }
    if (quad == 0 && lane == 0) RK_STAMP(grp, 0, 7);
  }
  tc_fence_before();
  return ok;
}

// ---- correction warps: O <- O * corr before the tile's P.V is added ---------------------------------------------
// One query tile of an item, whose O has not been written out yet.
struct Pending { int qt, bh; };

// O / l -> bf16 of one lane quadrant, through shared memory and TMA: a thread has a row, whose own stores would be one sector of a
// line each (3600 cycles from the softmax warps, which had nothing else to do then).
template <bool DUMP>
__device__ __forceinline__ void write_out_quadrant(const PrefillParams& p, const CUtensorMap* tmap_o, uint8_t* smem, uint32_t tmem_base, int g, int t_end,
                                                   const Pending& it) {
  using namespace c2;
  const int lane = threadIdx.x & 31;
  const int quad = (threadIdx.x >> 5) & 3;
  const int at = (g * 4 + (t_end & 3)) * 128 + quad * 32 + lane;
  const float inv_l = reinterpret_cast<const float*>(smem + corr_off)[at];
  const int row0 = it.qt * kBlockM + quad * 32;
  if (p.lse && row0 + lane < p.S_q) p.lse[(size_t)it.bh * p.S_q + row0 + lane] = reinterpret_cast<const float*>(smem + lse_off)[at];
  if (row0 >= p.S_q) return;      // no row of this quadrant exists: every chunk below commits a copy, which is what the wait for a half of the stage counts on
  uint8_t* stage = smem + stage_off + quad * 4096;
  tc_fence_after();
#pragma unroll 1
  for (int ch = 0; ch < p.d / 32; ++ch) {
    perturb<DUMP>(p, kPerturbOut, ch + quad);
    uint32_t r[32];
    tmem_ld32(tmem_base + (((uint32_t)(quad * 32)) << 16) + cO + g * 128 + ch * 32, r);
    tc_wait_ld();
    if (lane == 0) bulk_wait_read<1>();             // the copy that last left this half of the stage
    __syncwarp();
    uint8_t* dst = stage + (ch & 1) * 2048;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(r[8 * i + 2 * e]) * inv_l, __uint_as_float(r[8 * i + 2 * e + 1]) * inv_l);
        w[e] = *reinterpret_cast<const uint32_t*>(&b2);
      }
      *reinterpret_cast<uint4*>(dst + lane * 64 + ((i ^ ((lane >> 1) & 3)) * 16)) = make_uint4(w[0], w[1], w[2], w[3]);   // 64-byte swizzle
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) { tma_store_3d(tmap_o, dst, ch * 32, row0, it.bh); bulk_commit(); }
  }
  tc_fence_before();
}

// The tiles of one item; returns the code of the wait that gave up, or 0.  t0, t1: the two groups' tiles of earlier items.
template <bool DUMP, bool SPLIT>
__device__ __forceinline__ int correction_quadrant(const PrefillParams& p, const CUtensorMap* tmap_o, uint8_t* smem, uint64_t* bars, uint32_t tmem_base,
                                                   volatile int* abort_flag, int nt0, int nt1, int t0, int t1, const Pending& out0, const Pending& out1) {
  using namespace c2;
  const int lane = threadIdx.x & 31;
  const int quad = (threadIdx.x >> 5) & 3;
  const int row = quad * 32 + lane;
  const uint32_t lane_addr = ((uint32_t)(quad * 32)) << 16;
  const float* corr_sm = reinterpret_cast<const float*>(smem + corr_off);
  const int o_chunks = p.d / 32, n_all = max(nt0, nt1);
  for (int j = 0; j < n_all; ++j) {
    perturb<DUMP>(p, kPerturbCorr, j);
    if (stops<DUMP>(p, kPerturbCorr, j)) return 401;
#pragma unroll 1
    for (int g = 0; g < 2; ++g) {
      if (j >= (g == 0 ? nt0 : nt1)) continue;
      const int t = (g == 0 ? t0 : t1) + j;                   // this group's tile, counted over all items of the CTA
      if (quad == 0 && lane == 0) RK_STAMP(3, j, g * 4 + 0);
      if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bCF + (g * 4 + (t & 3)) * 4 + quad], (t >> 2) & 1, abort_flag))) return 401;
      const float corr = corr_sm[(g * 4 + (t & 3)) * 128 + row];
      if (quad == 0 && lane == 0) RK_STAMP(3, j, g * 4 + 1);
      if (t > 0) {
        // Always wait for the previous P.V of this tile, rescale or not: an arrival on the O-ready barrier then
        // implies that its previous phase has been consumed, which is what keeps the two-deep barrier from wrapping.
        if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bPV + g * 2 + ((t - 1) & 1)], ((t - 1) >> 1) & 1, abort_flag))) return 402;
      }
      if (j == 0) {
        if (!SPLIT && t > 0) write_out_quadrant<DUMP>(p, tmap_o, smem, tmem_base, g, t, g == 0 ? out0 : out1);   // the group's item before this one
      } else if (__any_sync(0xffffffffu, corr != 1.0f)) {
        tc_fence_after();
        if (quad == 0 && lane == 0) RK_STAMP(3, j, g * 4 + 2);
#pragma unroll 1
        for (int ch = 0; ch < o_chunks; ++ch) {
          uint32_t r[32];
          tmem_ld32(tmem_base + lane_addr + cO + g * 128 + ch * 32, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 2) mul2_ftz_inplace(r[i], r[i + 1], corr);
          tmem_st32(tmem_base + lane_addr + cO + g * 128 + ch * 32, r);
        }
        tc_wait_st();
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[bOR + g * 2 + (t & 1)]);   // the tile's P.V may accumulate into O now
      if (quad == 0 && lane == 0) RK_STAMP(3, j, g * 4 + 3);
    }
  }
  return 0;
}

// PREP: 64 columns (unit cu) of key tile `tile` of V, re-blocked along the keys by four warps (32 keys each), as TMA would have left them in their stage: rows of 128 bytes,
// 128-byte swizzle, zeros for keys that do not exist, and their part of the scale atom.  (Columns past d are left as they are: they meet columns of O that nobody reads.)
template <int FMT>
__device__ __forceinline__ void rebase_v_unit(const PrefillParams& p, uint8_t* smem, int warp, int lane, int st, int tile, int cu, int bhkv) {
  using namespace c2;
  const int quad = warp & 3, key0 = tile * kBlockN + quad * 32, n = max(0, min(32, p.S_kv - key0)), col = cu * 64 + (lane & 7) * 8;
  const int64_t row0 = (int64_t)bhkv * p.S_kv + (n > 0 ? key0 : 0);
  uint8_t* const dst = smem + v_off + st * kTileBytes + quad * 32 * 128;
  uint8_t* const atom = smem + sfv_off + st * kSfAtomBytes;
  uint32_t sc[2];
  auto at = [=](int k, int c) { return dst + k * 128 + (((c >> 4) ^ (k & 7)) << 4) + (c & 15); };
  rebase_block<FMT, 8, true, int>(p.v + row0 * p.d, p.v_sf + row0 * (p.d / 32), p.d, cu, n, reinterpret_cast<uint32_t (*)[32]>(smem + stage_off + warp * 256), lane,
                             [=](int k, const uint32_t (&o)[2]) { *reinterpret_cast<uint2*>(at(k, col)) = make_uint2(o[0], o[1]); },
                             [=](int k, int c, uint8_t code) { *at(k, col + c) = code; }, sc);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = col + (lane >> 3) * 2 + h;
    atom[sf_atom_offset(c, quad)] = (uint8_t)sc[h];
    if (p.d <= 64) atom[sf_atom_offset(c + 64, quad)] = 0x7F;
  }
}

// PREP: the scale atom of 128 rows from row0 of a matrix of S rows, by one warp, four rows a lane.
RK_DEVINL void scale_atom(const uint8_t* scales, int64_t bh, int S, int row0, int nbd, uint8_t* atom, int lane) {
  uint32_t w[4];
  row_scale_words(scales + (bh * S + row0 + lane) * nbd, scales, nbd, S - row0 - lane, nbd, w);
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<uint32_t*>(atom + sf_atom_offset(i * 32 + lane, 0)) = w[i];
}

template <bool SOFTCAP, bool DUMP, bool SPLIT, int PREP>
__global__ void __launch_bounds__(c2::kThreads, 1)
prefill2c_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const PrefillParams p, const uint32_t idesc_qk,
                 const uint32_t idesc_pv) {
  using namespace c2;
  extern __shared__ __align__(1024) uint8_t smem_raw2c[];
  uint8_t* smem = align_smem(smem_raw2c);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + bar_off);
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + misc_off + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) RK_STAMP(2, 0, 6);
  constexpr int kQt = SPLIT ? 1 : 2;                                  // query tiles per item
  constexpr bool kPrep = PREP >= 0, kPrepV = kPrep && PREP < kPrepScales;
  constexpr int kAtomTx = kPrep ? 0 : kSfAtomBytes;                   // of Q and K, by copy
  const int n_pairs = (p.n_q_tiles + kQt - 1) / kQt;
  auto decode = [&](uint32_t block) -> Work {
    Work w;
    const Place at = place_of_block(p, block, n_pairs);
    w.qp = at.index; w.bh = at.bh; w.bhkv = at.bhkv;
    int nt[2];                                                        // a tile past S_q needs none
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int qt = kQt * w.qp + g;
      nt[g] = (g < kQt && qt < p.n_q_tiles) ? key_tiles(p, qt) : 0;
    }
    // sliding window: key tiles wholly below the window of the pair's first row are masked for every row of both tiles
    w.j0 = 0;
    if (p.window > 0) {
      const int first_key = p.q_pos0 + kQt * w.qp * kBlockM - p.window + 1;  // lowest key the first row may see
      w.j0 = min(max(first_key, 0) / kBlockN, max(min(nt[0], nt[1] > 0 ? nt[1] : nt[0]) - 1, 0));
      nt[0] = max(nt[0] - w.j0, 0);                                       // tiles j0 .. j0 + nt - 1 are visited
      nt[1] = max(nt[1] - w.j0, 0);
    }
    w.nt0 = nt[0]; w.nt1 = nt[1];
    w.pad[0] = w.pad[1] = 0;
    return w;
  };
  Work w = {};

  auto issue_q = [&](int g) {
    uint64_t* bar = &bars[g == 0 ? bQ : bQB];
    mbar_arrive_expect_tx(bar, p.q_tile_tx + kAtomTx);
    tma_load_3d(smem + q_off + g * kTileBytes, &tmap_q, bar, 0, (kQt * w.qp + g) * kBlockM, w.bh);
    if (!kPrep) bulk_load_1d(smem + sfq_off + g * kSfAtomBytes, p.q_sf + ((size_t)w.bh * p.n_q_tiles + kQt * w.qp + g) * kSfAtomBytes, kSfAtomBytes, bar);
  };
  auto issue_kv = [&](int j, int st) {
    mbar_arrive_expect_tx(&bars[bKF + st], p.kv_tile_tx + kAtomTx);
    tma_load_3d(smem + k_off + st * kTileBytes, &tmap_k, &bars[bKF + st], 0, (j + w.j0) * kBlockN, w.bhkv);
    if (!kPrep) bulk_load_1d(smem + sfk_off + st * kSfAtomBytes, p.k_sf + ((size_t)w.bhkv * p.n_kv_tiles + j + w.j0) * kSfAtomBytes,
                 kSfAtomBytes, &bars[bKF + st]);
  };
  auto issue_v = [&](int j, int st) {
    mbar_arrive_expect_tx(&bars[bVF + st], p.kv_tile_tx + kAtomTx);
    const int key = (j + w.j0) * kBlockN;            // transposed V: [d][keys]
    tma_load_3d(smem + v_off + st * kTileBytes, &tmap_v, &bars[bVF + st], p.v_transposed ? key : 0, p.v_transposed ? 0 : key, w.bhkv);
    if (!kPrep) bulk_load_1d(smem + sfv_off + st * kSfAtomBytes, p.v_sf + ((size_t)w.bhkv * p.n_kv_tiles + j + w.j0) * kSfAtomBytes,
                 kSfAtomBytes, &bars[bVF + st]);
  };
  // The TMA warp sets up the barriers and goes on to its loads without waiting for the others, so that their latency runs under the
  // rest of the set-up.  Arrival counts: S-empty, P-full and O-ready take one arrival per warp of four.
  if (warp == kWarpTma) {
    for (int i = lane; i < nBars; i += 32) {
      const bool per_warp = (i >= bSE && i < bSE + 2) || (i >= bPF && i < bPF + 4) || (i >= bOR && i < bOR + 4);
      // SPLIT: both groups hand back S and write P, and the exchange takes a warp of each
      const bool both = SPLIT && (i < bPV || i >= bCF + 16) && i < bOR;
      mbar_init(&bars[i], per_warp ? (both ? 8 : 4) : both && i >= bCF + 16 ? 2 : i == bWE ? kReaders : kPrep && i >= bVF && i < bVF + kStages ? (!kPrepV ? 2 : p.d > 64 ? 8 : 4) : kPrep && i == bPrep ? 3 : 1);
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
    if (SPLIT && work_par) return 0;
    if (!__all_sync(0xffffffffu, mbar_wait_compact(&bars[bWF], work_par, abort_flag))) return -1;
    work_par ^= 1;
    w = *reinterpret_cast<const Work*>(smem + work_off);
    if (w.qp < 0) return 0;
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars[bWE]);
    return 1;
  };
  constexpr int kFailWork = 501;

  if constexpr (kPrep) {
    w = decode(blockIdx.x);
    if (warp > kWarpTma) {
      // Atoms of Q and of the key tiles by the three warps that have nothing to do before these are there.  (By one of them, atom after atom or all loads at once: one head of 256
      // keys 2 us more.)
#pragma unroll 1
      for (int a = warp - kWarpTma - 1; a <= w.nt0 && w.nt0 > 0; a += 3) {
        perturb<DUMP>(p, kPerturbAtoms, a);
        scale_atom(a == 0 ? p.q_sf : p.k_sf, a == 0 ? w.bh : w.bhkv, a == 0 ? p.S_q : p.S_kv, a == 0 ? w.qp * kBlockM : (a - 1 + w.j0) * kBlockN, p.d / 32,
                   smem + (a == 0 ? sfq_off : sfk_off + (a - 1) * kSfAtomBytes), lane);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && !stops<DUMP>(p, kPerturbAtoms, warp - kWarpTma - 1)) mbar_arrive(&bars[bPrep]);
    } else if (!kPrepV) {
      if (warp < w.nt0 && __shfl_sync(0xffffffffu, lane == 0 ? *reinterpret_cast<volatile int*>(p.status) : 0, 0) == 0) {      // V's scales: a warp per key tile
        const int nkb = (p.S_kv + 31) / 32, block = (warp + w.j0) * 4;
        uint32_t words[4];
        perturb<DUMP>(p, kPerturbV, warp);
        key_scale_words(p.v_sf + ((int64_t)w.bhkv * nkb + block) * p.d + lane * 4, p.d, nkb - block, lane * 4 < p.d, (reinterpret_cast<uintptr_t>(p.v_sf) & 3) == 0, words);
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint32_t*>(smem + sfv_off + warp * kSfAtomBytes + sf_atom_offset(lane * 4 + i, 0)) = words[i];
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && !stops<DUMP>(p, kPerturbV, warp + 2 - w.nt0)) mbar_arrive(&bars[bVF + warp]);
      }
    } else if (warp < kWarpTma) {
      // V, by the twelve warps that have nothing to do before the first scores are there: units of 64 columns, in the order of the tiles; the correction warps, which are needed last, take
      // the fourth as well.  Where an earlier launch gave up V does not come, and O is not written.
      const int units = p.d > 64 ? 2 : 1, n = w.nt0 * units, grp = warp >> 2;
      if (__shfl_sync(0xffffffffu, lane == 0 ? *reinterpret_cast<volatile int*>(p.status) : 0, 0) == 0) {
#pragma unroll 1
        for (int i = grp; i < n; i += grp == 2 ? (i == 2 ? 1 : n) : 4) {
          const int st = units == 2 ? i >> 1 : i;
          perturb<DUMP>(p, kPerturbV, i);
          rebase_v_unit<kPrepV ? PREP : 0>(p, smem, warp, lane, st, st + w.j0, units == 2 ? i & 1 : 0, w.bhkv);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && !stops<DUMP>(p, kPerturbV, warp & 3)) mbar_arrive(&bars[bVF + st]);
        }
      }
    }
  }
  // (The softmax branch comes last in the code: measured 1-1.5 % faster than first.)
  if (warp >= kWarpTma) {
    reg_dec<SPLIT ? kRegIssueSplit : kRegIssue>();
    int fail = 0;                                    // which wait gave up
    // before TMEM and shared memory go back: this thread's asynchronous work has finished, also where the CTA gives up
    auto drain = [&](uint64_t* bar, uint32_t parity, int code) { if (!mbar_wait_short<true>(bar, parity, nullptr) && !fail) fail = code; };
    if (threadIdx.x == kWarpQk * 32) RK_STAMP_RAW(6);
    if (warp == kWarpTma) {
      // ================= TMA producer; hands out the items =================
      if (lane == 0) {
        prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
        int stopped = 0, st = 0, q_used = 0, q_par = 0;
        uint32_t use = 0, block = blockIdx.x;
        for (uint32_t k = 0;; ++k) {
          w = decode(block);
          const int n_all = max(w.nt0, w.nt1);
          for (int j = 0; j < n_all || j == 0; ++j) {
            perturb<DUMP>(p, kPerturbTma, j);
            if (stops<DUMP>(p, kPerturbTma, j)) { fail = 201; break; }
            if (j == 0) {
              // everybody has read the last item: this one takes its place
              if (k > 0 && !mbar_wait_compact<true>(&bars[bWE], (k - 1) & 1, abort_flag)) { fail = 502; break; }
              *reinterpret_cast<Work*>(smem + work_off) = w;
              mbar_arrive(&bars[bWF]);
              if (k == 0) {
                grid_dependency_wait();
                stopped = *reinterpret_cast<volatile int*>(p.status);       // an earlier launch gave up on a wait
              }
#pragma unroll 1
              for (int g = 0; g < 2; ++g) {
                if ((g == 0 ? w.nt0 : w.nt1) == 0) continue;
                if ((q_used >> g) & 1) {             // Q K^T of the last item that had a tile in this place has finished
                  if (!mbar_wait_compact<true>(&bars[bQE + g], (q_par >> g) & 1, abort_flag)) { fail = 203; break; }
                  q_par ^= 1 << g;
                }
                q_used |= 1 << g;
                issue_q(g);
              }
              if (fail) break;
            }
            if (n_all > 0) {
              if (use > 0 && !mbar_wait_compact<true>(&bars[bKE + st], (use - 1) & 1, abort_flag)) { fail = 201; break; }
              issue_kv(j, st);
              if (stopped) break;                    // O is written only where V has come
              if (kPrepV) { ++st; continue; }        // (a stage for every tile)
              if (use > 0 && !mbar_wait_compact<true>(&bars[bVE + st], (use - 1) & 1, abort_flag)) { fail = 202; break; }
              issue_v(j, st);
              if (++st == kStages) { st = 0; ++use; }
            }
          }
          if (stopped) *abort_flag = kStopped;
          if (fail || stopped || SPLIT) break;
          // The next item is asked for now that this one's last loads are under way, three tiles before its end, and not earlier: the items
          // that are left go to the SMs that are free first.
          mbar_arrive_expect_tx(&bars[bClc], 16);
          clc_request(smem + clc_off, &bars[bClc]);
          drain(&bars[bClc], k & 1, 503);
          if (fail) break;
          if (!clc_answer(smem + clc_off, block)) {
            if (!mbar_wait_compact<true>(&bars[bWE], k & 1, abort_flag)) { fail = 502; break; }
            w.qp = -1;
            *reinterpret_cast<Work*>(smem + work_off) = w;
            mbar_arrive(&bars[bWF]);
            break;
          }
          fence_proxy_async_smem();                  // the answer has been read before the next one may overwrite it
        }
        // The last loads into each place have arrived, also those whose readers have given up (this lane alone starts phases of these barriers).
        // One wait in a loop over a bit mask: with a wait each for K, V and Q the kernel was 0.6 % slower, by the mere size of the code.
        const bool k_ahead = fail == 202 || (stopped && q_used);      // K of a tile has been asked for, V has not
        uint32_t want = q_used & 1, par = q_par & 1;                  // bits: barrier indices, bQBit for group B's Q
        constexpr int bQBit = bVF + kStages;
        static_assert(bQ == 0 && bQBit < 32, "one word");
        if (q_used >> 1) { want |= 1u << bQBit; par |= (uint32_t)(q_par >> 1) << bQBit; }
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
          const uint32_t nv = use + (i < st), nk = nv + (i == st && k_ahead);      // loads into this stage
          want |= (uint32_t)(nk > 0) << (bKF + i) | (uint32_t)(nv > 0 && !kPrepV) << (bVF + i);
          par |= ((nk - 1) & 1) << (bKF + i) | ((nv - 1) & 1) << (bVF + i);
        }
#pragma unroll 1
        for (; want; want &= want - 1) {
          const int b = __ffs(want) - 1;
          drain(&bars[b == bQBit ? bQB : b], (par >> b) & 1, 301);
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
      int st = 0;
      uint32_t use_par = 0;                    // K stage of the tile and the parity of its use
      uint32_t q_par = 0, t_par = 0;           // bit g: parities of group g's next Q tile and of its next key tile
      int last_g = -1;                         // which group read the shared S columns last, and at which tile parity
      uint32_t last_par = 0;
      for (int more; (more = warp_uniform(next_work())) != 0;) {
        if (more < 0) { fail = kFailWork; break; }
        const int nt0 = warp_uniform(w.nt0), nt1 = warp_uniform(w.nt1), n_all = max(nt0, nt1);
        for (int j = 0; j < n_all && !fail; ++j) {
          perturb<DUMP>(p, kPerturbQk, j);
          if (stops<DUMP>(p, kPerturbQk, j)) { fail = 302; break; }
          if (lane == 0) RK_STAMP(2, j, 0);
          if (kPrep && j == 0 && !__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bPrep], 0, abort_flag))) { fail = 309; break; }
          if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bKF + st], use_par, abort_flag))) { fail = 302; break; }
          if (elect_one()) tc_cp_32x128b_warpx4(tm + cSfK + st * 4, dsfk + (uint32_t)(st * (kSfAtomBytes >> 4)));
          const uint64_t dkt = dk + (uint32_t)(st * (kTileBytes >> 4));
          if (lane == 0) RK_STAMP(2, j, 1);
          // rolled on purpose: this warp shares the instruction cache with the softmax warps (both groups unrolled, 8 x 16 heads of 4096:
          // 524 -> 540 us, the P V issuer's as well 560; the four MMAs rolled too 521.3 -> 519.4, those of P V no gain)
#pragma unroll 1
          for (int g = 0; g < 2; ++g) {
            const int n_mine = g == 0 ? nt0 : nt1;
            if (j >= n_mine) continue;
            if (j == 0) {
              if (!__all_sync(0xffffffffu, mbar_wait_compact(&bars[g == 0 ? bQ : bQB], (q_par >> g) & 1, abort_flag))) { fail = 301; break; }
              q_par ^= 1u << g;
              if (elect_one()) tc_cp_32x128b_warpx4(tm + cSfQ + g * 4, dsfq + (uint32_t)(g * (kSfAtomBytes >> 4)));
            }
            if (last_g >= 0 && !__all_sync(0xffffffffu, mbar_wait_compact(&bars[bSE + last_g], last_par, abort_flag))) { fail = 305; break; }
            tc_fence_after();
            const uint64_t dqt = dq + (uint32_t)(g * (kTileBytes >> 4));
            if (elect_one()) {
#pragma unroll 1
              for (int kk = 0; kk < 4; ++kk)
                mma_mxf8f6f4_ss(tm + cS, dqt + kk * 2, dkt + kk * 2, idesc_with_sf(idesc_qk, kk, kk), tm + cSfQ + g * 4, tm + cSfK + st * 4, kk > 0 ? 1u : 0u);
              tc_commit(&bars[bSF + g]);
              if (!SPLIT && j == n_mine - 1) tc_commit(&bars[bQE + g]);
              if (j >= (g == 0 ? nt1 : 0)) tc_commit(&bars[bKE + st]);      // the last group with this tile
            }
            last_g = g; last_par = (t_par >> g) & 1;
            t_par ^= 1u << g;
            if (lane == 0) RK_STAMP(2, j, 2 + g);
          }
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
      int st = 0, t0 = 0, t1 = 0;              // t0, t1: the groups' key tiles of earlier items
      uint32_t use_par = 0;
      for (int more; (more = warp_uniform(next_work())) != 0;) {
        if (more < 0) { fail = kFailWork; break; }
        const int nt0 = warp_uniform(w.nt0), nt1 = warp_uniform(w.nt1), n_all = max(nt0, nt1);
        for (int i = 0; i < n_all && !fail; ++i) {
          perturb<DUMP>(p, kPerturbPv, i);
          if (stops<DUMP>(p, kPerturbPv, i)) { fail = 303; break; }
          if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bVF + st], use_par, abort_flag))) { fail = 303; break; }
          if (elect_one()) tc_cp_32x128b_warpx4(tm + cSfV + st * 4, dsfv + (uint32_t)(st * (kSfAtomBytes >> 4)));
          const uint64_t dvt = dv + (uint32_t)(st * (kTileBytes >> 4));
#pragma unroll 1
          for (int g = 0; g < 2; ++g) {
            if (i >= (g == 0 ? nt0 : nt1)) continue;
            const int t = (g == 0 ? t0 : t1) + i, gb = g * 2 + (t & 1);
            const uint32_t par2 = (t >> 1) & 1;
            if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bPF + gb], par2, abort_flag))) { fail = 304; break; }      // P written
            if (!__all_sync(0xffffffffu, mbar_wait_compact<true>(&bars[bOR + gb], par2, abort_flag))) { fail = 307; break; }      // O rescaled for this tile, or the last item's written out
            tc_fence_after();
            const uint64_t dpt = dp + (uint32_t)(gb * (kTileBytes >> 4));
            if (elect_one()) {
              tc_cp_32x128b_warpx4(tm + cSfP + gb * 4, dsfp + (uint32_t)(gb * (kSfAtomBytes >> 4)));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                mma_mxf8f6f4_ss(tm + cO + g * 128, dpt + kk * 2, dvt + kk * v_kk, idesc_with_sf(idesc_pv, kk, kk), tm + cSfP + gb * 4, tm + cSfV + st * 4,
                                (i > 0 || kk > 0) ? 1u : 0u);
              tc_commit(&bars[bPV + gb]);
              if (i >= (g == 0 ? nt1 : 0)) tc_commit(&bars[bVE + st]);      // the last group with this tile
            }
            if (lane == 0) RK_STAMP(2, i, 4 + g);
          }
          if (++st == kStages) { st = 0; use_par ^= 1; }
        }
        if (fail) break;
        t0 += nt0; t1 += nt1;
      }
      if (elect_one()) tc_commit(&bars[bDRAIN2]);
      drain(&bars[bDRAIN2], 0, 308);
      __syncwarp();
    }
    if (fail) give_up(abort_flag, p.status, fail);
  } else if (warp >= kWarpCorr) {
    reg_dec<SPLIT ? kRegCorrSplit : kRegCorr<SOFTCAP>>();
    int t0 = 0, t1 = 0, fail = 0;                    // t0, t1: the groups' key tiles of earlier items
    Pending out0{0, 0}, out1{0, 0};
    for (;;) {
      const int more = next_work();
      if (more < 0) { fail = kFailWork; break; }
      if (more == 0 && SPLIT) break;
      if (more == 0) { w.nt0 = t0 > 0; w.nt1 = t1 > 0; }      // no item is left: once more, for the O of the last ones
      fail = correction_quadrant<DUMP, SPLIT>(p, &tmap_o, smem, bars, tmem_base, abort_flag, w.nt0, w.nt1, t0, t1, out0, out1);
      if (fail || more == 0) break;
      t0 += w.nt0; t1 += w.nt1;
      if (w.nt0 > 0) out0 = Pending{2 * w.qp, w.bh};
      if (w.nt1 > 0) out1 = Pending{2 * w.qp + 1, w.bh};
    }
    if (!SPLIT && lane == 0) bulk_wait_all();
    if (fail) give_up(abort_flag, p.status, fail);
  } else {
    reg_inc<SPLIT ? kRegSoftmaxSplit : kRegSoftmax<SOFTCAP>>();
    if (threadIdx.x == 0) RK_STAMP_RAW(5);
    const int grp = warp >> 2;
    int t0 = 0;                                      // this group's key tiles of earlier items
    for (int more; (more = next_work()) != 0;) {
      if (more < 0) { give_up(abort_flag, p.status, kFailWork); break; }
      const int qt = SPLIT ? w.qp : 2 * w.qp + grp, n_mine = SPLIT || grp == 0 ? w.nt0 : w.nt1;
      if (n_mine > 0) {
        if (!softmax_row_group<SOFTCAP, DUMP, SPLIT>(p, smem, bars, tmem_base, abort_flag, grp, qt, w.bh, n_mine, w.j0, t0)) break;
        t0 += n_mine;
      } else if (qt < p.n_q_tiles && !(SPLIT && grp == 1)) {
        // no visible key: O = 0 (the l <= 0 guard of finalize_O, kernels/flash_attention_mx_gemma/flash_mx_impl.hpp:554-560)
        const int q_row = qt * kBlockM + (int)(threadIdx.x & 127);
        if (q_row < p.S_q && *reinterpret_cast<volatile int*>(p.status) == 0) {
          __nv_bfloat16* orow = p.o + ((size_t)w.bh * p.S_q + q_row) * p.d;
#pragma unroll 1
          for (int c = 0; c < p.d; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
          if (p.lse) p.lse[(size_t)w.bh * p.S_q + q_row] = __int_as_float(0xff800000);
        }
      }
    }
    if (!SPLIT && t0 > 0) {                          // the last item's O may be written out
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[bCF + (grp * 4 + (t0 & 3)) * 4 + (warp & 3)]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) RK_STAMP(2, 0, 7);
  if (warp == kWarpQk) { tc_fence_after(); tmem_dealloc(tmem_base, kTmemCols); }
}

template <bool SOFTCAP, bool DUMP, bool SPLIT, int PREP = -1>
static int launch2c_cfg(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                        uint32_t idesc_qk, uint32_t idesc_pv, cudaStream_t st) {
  const int smem_bytes = c2::total + 1024;
  const dim3 grid((SPLIT ? p.n_q_tiles : (p.n_q_tiles + 1) / 2) * p.H * p.B);
  auto kern = prefill2c_kernel<SOFTCAP, DUMP, SPLIT, PREP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess) return (int)e;
  if (g_ev_before && g_ev_after) cudaEventRecord(g_ev_before, st);
  e = launch_pdl(kern, grid, dim3(c2::kThreads), smem_bytes, st, tq, tk, tv, to, p, idesc_qk, idesc_pv);
  if (g_ev_before && g_ev_after) cudaEventRecord(g_ev_after, st);
  return (int)e;
}

int launch_prefill2c(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                     uint32_t idesc_qk, uint32_t idesc_pv, bool softcap, bool split, int prep, cudaStream_t st) {
  if (prep == c2::kPrepScales)
    return p.dbg || p.perturb ? launch2c_cfg<false, true, true, c2::kPrepScales>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                              : launch2c_cfg<false, false, true, c2::kPrepScales>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st);
  if (prep >= 0) {
    if (p.dbg || p.perturb) return prep == RK_FMT_E4M3 ? launch2c_cfg<false, true, true, RK_FMT_E4M3>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                                                       : launch2c_cfg<false, true, true, RK_FMT_E5M2>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st);
    return prep == RK_FMT_E4M3 ? launch2c_cfg<false, false, true, RK_FMT_E4M3>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                               : launch2c_cfg<false, false, true, RK_FMT_E5M2>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st);
  }
  if (p.dbg || p.perturb)      // the tests' stage dump and delays live in instantiations of their own: the kernels that ship carry none of their code
    return split ? (softcap ? launch2c_cfg<true, true, true>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                            : launch2c_cfg<false, true, true>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st))
                 : (softcap ? launch2c_cfg<true, true, false>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                            : launch2c_cfg<false, true, false>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st));
  return split ? (softcap ? launch2c_cfg<true, false, true>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                          : launch2c_cfg<false, false, true>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st))
               : (softcap ? launch2c_cfg<true, false, false>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st)
                          : launch2c_cfg<false, false, false>(tq, tk, tv, to, p, idesc_qk, idesc_pv, st));
}

}  // namespace rk
