// Definitions shared by the prefill kernels (d = 256; d <= 128: pairs of query tiles, and one at a time).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "rk_common.cuh"
#include "rk_internal.h"

namespace rk {

constexpr int kBlockM = 128;
constexpr int kBlockN = 128;
constexpr int kTileBytes = 128 * 128;      // one [128 rows][128 B] swizzled tile
constexpr int kSfAtomBytes = 512;
constexpr uint32_t kTmemCols = 512;

// TMEM column map
constexpr uint32_t kColS = 0;
constexpr uint32_t kColO = 128;
constexpr uint32_t kColSfQ = 384;                 // + ch*4
constexpr uint32_t kColSfK = 392;                 // + stage*8 + ch*4   (<= 3 stages)
constexpr uint32_t kColSfP = 416;                 // + pbuf*4
constexpr uint32_t kColSfV = 424;                 // + stage*8 + ch*4

struct PrefillParams {
  const uint8_t* q_sf;
  const uint8_t* k_sf;
  const uint8_t* v_sf;
  const uint8_t* v;    // a call whose attention kernel does the preparation: V's codes, and q_sf, k_sf, v_sf as the caller gave them
  __nv_bfloat16* o;
  float* lse;
  int* status;
  float* dbg;          // optional stage dump (tests): last query tile of the first head, first key tile
  int B, H, H_kv, S_q, S_kv, d;
  int group;           // query heads per KV head
  int n_q_tiles, n_kv_tiles;
  int head_group;      // (batch, head) pairs per work-order group: the heaviest query tiles of a whole group run first
  int q_pos0, causal, window;
  int q_tile_tx, kv_tile_tx;   // bytes one Q / K / V tile load adds to its mbarrier: 16384, 12288 for 6-bit, 8192 for 4-bit tensors
                               // (the transaction counts the packed source bytes, not the padded shared-memory image)
  int v_transposed;    // V tiles are [d][keys] (K-major B operand; 6-bit V) instead of [keys][d]
  int perturb;         // test hook: warp role that sleeps a little at every key tile, or kStopRole + one that gives up (0 = none)
  float scale_log2;    // softmax_scale * log2(e)
  float cap_log2;      // softcap * log2(e)
  float inv_cap_scale; // softmax_scale / softcap
};

// Value of a CTA's abort flag where an earlier launch gave up on a wait and this one does nothing (its waits end, and nothing is reported).
constexpr int kStopped = 2;
RK_DEVINL void give_up(volatile int* abort_flag, int* status, int code) {
  if (*abort_flag != kStopped) report_wait_failure(abort_flag, status, code);
}

// Registers moved between warpgroups.
template <uint32_t N> RK_DEVINL void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <uint32_t N> RK_DEVINL void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// Work order over the block indices: (batch, head) pairs are taken in groups of p.head_group; inside a group the heaviest (latest) of the n places
// of a head -- query tiles, or pairs of them -- come first for all its heads and the lightest last, so the grid ends on short items, while a
// group's K/V still fits in L2.
struct Place { int index, bh, bhkv; };      // place within the head, b * H + h, b * H_kv + h / group
RK_DEVINL Place place_of_block(const PrefillParams& p, uint32_t block, int n) {
  const uint32_t n_bh = p.B * p.H, per_group = n * p.head_group;
  const uint32_t grp_i = block / per_group, r = block - grp_i * per_group;
  const uint32_t heads_here = min((uint32_t)p.head_group, n_bh - grp_i * p.head_group);
  const uint32_t down = r / heads_here;
  Place w;
  w.index = n - 1 - (int)down;
  w.bh = grp_i * p.head_group + (r - down * heads_here);
  w.bhkv = (uint32_t)w.bh / (uint32_t)p.group;
  return w;
}
// Key tiles a query tile needs, from the first: causal tiles wholly above the diagonal are never touched (blocks_used,
// kernels/flash_attention_mx_gqa/flash_attention_model.py:182-186).
RK_DEVINL int key_tiles(const PrefillParams& p, int qt) {
  if (!p.causal) return p.n_kv_tiles;
  const int max_qpos = p.q_pos0 + min(qt * kBlockM + kBlockM, p.S_q) - 1;
  return max_qpos < 0 ? 0 : min(p.n_kv_tiles, max_qpos / kBlockN + 1);
}

// Test hooks, in the instantiations for tests alone.  perturb: the role sleeps a little, longer or shorter from key tile to key tile.
template <bool DUMP>
RK_DEVINL void perturb(const PrefillParams& p, int role, int j) {
  if (DUMP && __builtin_expect(p.perturb == role, 0)) __nanosleep(400 + 97 * (j & 7));
}
// stops: the role acts as if its wait had run out, at its first key tile that is not an item's first.
constexpr int kStopRole = 100;
template <bool DUMP>
RK_DEVINL bool stops(const PrefillParams& p, int role, int j) { return DUMP && p.perturb == kStopRole + role && j >= 1; }

// 32 bytes of a row of O by one thread: a whole sector in one store where O is 32-byte aligned (rows are multiples of 64 bytes), where two stores of
// a thread with a row of its own are half a sector each (d = 256, 2 x 16/8 heads of 8192, under the power cap: 969 -> 958 us); O is guaranteed to be
// 16-byte aligned only.
RK_DEVINL void store_row32(__nv_bfloat16* dst, const uint32_t (&w)[8], bool aligned32) {
  if (aligned32) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
  } else {
    reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

RK_DEVINL float fmax3(float a, float b, float c) { float d; asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c)); return d; }
// packed fp32 pairs (two lanes per instruction on the FMA pipe)
RK_DEVINL void mul2_ftz_inplace(uint32_t& a0, uint32_t& a1, float b) {                 // a *= b on two fp32 bit patterns, in their registers
  asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%0, %1};\n\tmov.b64 rb, {%2, %2};\n\tmul.rn.ftz.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
      : "+r"(a0), "+r"(a1) : "f"(b));
}
// Packed operations on values that stay in 64-bit registers (two fp32 lanes each): a broadcast operand is
// packed once by the caller instead of once per instruction.
RK_DEVINL uint64_t pack2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
RK_DEVINL void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
RK_DEVINL void unpack2u(uint64_t v, uint32_t& lo, uint32_t& hi) { asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v)); }
RK_DEVINL uint64_t fma2p(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
RK_DEVINL uint64_t add2p(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
RK_DEVINL uint64_t mul2p_ftz(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
// Soft cap of two scores in the log2 domain: cap_log2 * tanh(s * scale / cap), tanh(y) = 1 - 2 / (1 + e^(2y)).
// The exponential is the one special-function instruction; the reciprocal is three Newton steps on the FMA pipe from
// an integer first guess (error 0.12 -> 1.4e-2 -> 2e-4 -> 4e-8), because the special-function unit is what bounds
// the capped kernels (it also has the softmax exponential to do).  k2 = 2 log2(e) scale / cap; the exponent is
// clamped so that 1 + e stays finite (by a minimum that lets NaN through, as the series does).
RK_DEVINL float fmin_nan(float a, float b) { float d; asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b)); return d; }
RK_DEVINL void softcap_pair(float& s0, float& s1, float k2, uint64_t one2, uint64_t m2cap2, uint64_t cap2) {
  const float e0 = ex2_approx(fmin_nan(s0 * k2, 126.0f)), e1 = ex2_approx(fmin_nan(s1 * k2, 126.0f));
  const uint64_t z = add2p(pack2(e0, e1), one2);                       // 1 + e in [1, 2^126]
  uint32_t z0, z1;
  unpack2u(z, z0, z1);
  uint64_t r = pack2(__uint_as_float(0x7EF311C7u - z0), __uint_as_float(0x7EF311C7u - z1));
  const uint64_t nz = z ^ 0x8000000080000000ull;                       // -z
#pragma unroll
  for (int it = 0; it < 3; ++it) r = fma2p(r, fma2p(nz, r, one2), r);   // r += r * (1 - z r)
  unpack2(fma2p(r, m2cap2, cap2), s0, s1);                              // cap_log2 * (1 - 2 r)
}

RK_DEVINL float fabsmax3(float a, float b, float c) { float d; asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c)); return d; }
RK_DEVINL uint64_t mul2p(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// The soft cap of a whole set of scores, in place: s <- cap_log2 * tanh(s * scale / cap).
// While every |s * scale / cap| of a warp's scores is at most 1/8 (logits of a model that caps at 50 are two orders
// of magnitude below that) tanh is its series y - y^3/3 + 2 y^5/15 - 17 y^7/315 (next term below 1.4e-9 of y),
// evaluated in s^2 with the constants folded into the coefficients: five packed FMA-pipe operations per pair of
// scores and no special-function operation, against an exponential and a Newton reciprocal per score in
// softcap_pair, which is kept for the scores that are not small.  The decision is per warp and 64 keys of a key tile, whether a thread has
// 64 scores of the tile or all 128: the two forms differ in a score's last bits, and a row comes out the same in every form of the kernels.
// Both sets of a thread with 128 are decided by one reduction over the warp, and the series of both is one run of code, against two votes and a
// branch for each: 8 x 16 heads of 4096 at d = 128, cap 50, 810 us and 784; decided for all 128 at once 791. (Logits of standard deviation 4, all
// exponential: 1 242, 1 247 and 1 206.)
template <int N>
RK_DEVINL void softcap_scores(float (&s)[N], float scale_log2, float cap_log2, float inv_cap_scale) {
  static_assert(N == 64 || N == 128, "one or two sets of 64 scores");
  auto is_small = [&](const int h) -> uint32_t {
    float b0 = fabsmax3(s[h], s[h + 1], s[h + 2]), b1 = fabsmax3(s[h + 3], s[h + 62], s[h + 63]);
#pragma unroll
    for (int c = h + 4; c < h + 60; c += 4) { b0 = fabsmax3(b0, s[c], s[c + 1]); b1 = fabsmax3(b1, s[c + 2], s[c + 3]); }
    b0 = fabsmax3(b0, s[h + 60], s[h + 61]);
    return fmaxf(b0, b1) * inv_cap_scale <= 0.125f ? 1u : 0u;           // 0 where all are NaN
  };
  auto series = [&](const int from, const int to) {
    const float q = inv_cap_scale * inv_cap_scale;
    const float c1 = -0.3333333333f * q * scale_log2, c2 = 0.1333333333f * q * q * scale_log2,
                c3 = -0.05396825397f * q * q * q * scale_log2;
    const uint64_t k1 = pack2(c1, c1), k2 = pack2(c2, c2), k3 = pack2(c3, c3), a2 = pack2(scale_log2, scale_log2);
#pragma unroll
    for (int c = from; c < to; c += 2) {
      const uint64_t v = pack2(s[c], s[c + 1]);
      const uint64_t z = mul2p(v, v);
      uint64_t t = fma2p(z, k3, k2);
      t = fma2p(z, t, k1);
      t = fma2p(z, t, a2);
      unpack2(mul2p(v, t), s[c], s[c + 1]);
    }
  };
  auto exponential = [&](const int from, const int to) {
    const float k2 = 2.0f * 1.4426950408889634f * inv_cap_scale;
    const uint64_t one2 = pack2(1.0f, 1.0f), m2cap2 = pack2(-2.0f * cap_log2, -2.0f * cap_log2), cap2 = pack2(cap_log2, cap_log2);
#pragma unroll
    for (int c = from; c < to; c += 2) softcap_pair(s[c], s[c + 1], k2, one2, m2cap2, cap2);
  };
  constexpr uint32_t kAll = N == 64 ? 1 : 3;                            // one bit per set
  uint32_t small = is_small(0);
  if (N == 128) small = __reduce_and_sync(0xffffffffu, small + 2 * is_small(N - 64));
  else small = __all_sync(0xffffffffu, small) ? 1u : 0u;
  if (small == kAll) series(0, N);
  else if (N == 64) exponential(0, N);
  else {
    if (small == 1) series(0, 64);
    if (small == 2) series(N - 64, N);
    if (!(small & 1)) exponential(0, 64);
    if (!(small & 2)) exponential(N - 64, N);
  }
}

// two ints (0..255 each) into bytes 1:0 of the result, bytes 3:2 taken from the low half of c
RK_DEVINL uint32_t pack_u8x2(uint32_t hi, uint32_t lo, uint32_t c) {
  uint32_t d; asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(c)); return d;
}

RK_DEVINL float ld_shared_f32(const float* p) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(smem_u32(p)) : "memory"); return v; }
// The same behind the answer of a barrier test, and only where it was yes; `otherwise` where not.  A load that does not depend on the answer can be served before the test is and
// bring what was there before, beside a yes: with a role delayed (the tests' hook), d = 256, 74 heads of 700 keys with a window of 150, one call in six had rows of O
// rescaled by a maximum of four tiles ago.
RK_DEVINL float ld_shared_f32_if(bool yes, const float* p, float otherwise) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.shared.f32 %0, [%1];\n\t}" : "+f"(otherwise) : "r"(smem_u32(p)), "r"((uint32_t)yes) : "memory");
  return otherwise;
}

#ifdef RK_X_STAMPS
// Timeline stamps (measurement builds of the d <= 128 kernel only): clock64 of chosen events of one CTA, written into the dump buffer, by role and key
// tile of an item.  A CTA that takes several items leaves those of the last one that had the tile.
// The CTA is RK_X_STAMP_BLOCK, or the block index b when the perturbation hook is set to 1000 + b.
#ifndef RK_X_STAMP_BLOCK
#define RK_X_STAMP_BLOCK 0
#endif
#define RK_STAMP_CTA ((int)blockIdx.x == (p.perturb >= 1000 ? p.perturb - 1000 : RK_X_STAMP_BLOCK))
#define RK_STAMP(slot, j, k) do { if (p.dbg && RK_STAMP_CTA && (j) < 32) \
    reinterpret_cast<unsigned*>(p.dbg)[24576 + (slot) * 512 + (j) * 8 + (k)] = (unsigned)clock64(); } while (0)
#define RK_STAMP_RAW(idx) do { if (p.dbg && RK_STAMP_CTA) \
    reinterpret_cast<unsigned*>(p.dbg)[24576 + 2048 + (idx)] = (unsigned)clock64(); } while (0)
#else
#define RK_STAMP(slot, j, k) do {} while (0)
#define RK_STAMP_RAW(idx) do {} while (0)
#endif


int make_tmap_u8_3d(CUtensorMap* m, const void* base, int64_t BH, int64_t S, int64_t d);
int make_tmap_sub8_3d(CUtensorMap* m, const void* base, int64_t BH, int64_t rows, int64_t cols_padded, int bits);
extern float* g_prefill_dbg;

// Two query tiles per CTA, one thread per row, correction warps (d <= 128), or with `split` one query tile; defined in rk_prefill2c.cu.
int launch_prefill2c(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                     uint32_t idesc_qk, uint32_t idesc_pv, bool softcap, bool split, int prep, cudaStream_t st);
// One query tile per CTA at a time, two softmax groups on alternate key tiles (d <= 128, few query tiles); defined in rk_prefill1.cu.
int launch_prefill1(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                    uint32_t idesc_qk, uint32_t idesc_pv, bool softcap, cudaStream_t st);
extern int g_prefill_perturb;   // test hook: PrefillParams::perturb of the next launches
extern int g_prefill_form;      // test hook: the form of the next launches at d <= 128, 0 = by prefill_form

}  // namespace rk
