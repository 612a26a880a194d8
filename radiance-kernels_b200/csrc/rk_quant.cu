// MX block quantizer kernels (HBM-bound streaming kernels, no tensor cores).
//
//  quantize_rows   fp32 [rows][cols] -> codes + one E8M0 scale per 32 contiguous
//                  elements.  Same results as quantize_one_block,
//                  kernels/simt_quant/kernel.cpp:95-129 (golden:
//                  lib/golden/golden.py:118-170), bit for bit.  4 lanes share a
//                  block, each lane loads 2 x float4 and stores 8 packed codes.
//                  Algorithmic traffic 4 B in + 1 B + 1/32 B out per element.
//  quantize_keys   same rule with the blocks running down the rows (the key
//                  axis) of each matrix in a batch -- the reference's V layout
//                  (kernels/flash_attention_mx/gen_data.py:77).
//  rebase_v        codes+scales blocked along d -> decode exactly -> re-block
//                  along the keys.  Writes the scales either row-major
//                  [ceil(S/32)][d] or directly in the 512-byte scale-factor
//                  atoms the attention kernel copies into TMEM.
//  retile_scales   block scales in the other layouts -> scale-factor atoms.
//
// Element encoding: the reference's integer round-shift encoder (rk::encode_rne)
// defines the result.  The hot loops use the hardware converter
// cvt.rn.satfinite.<fmt>x2.f32 instead, which verify_encoder_kernel proves equal
// to it on every finite fp32 input (all 2^32 bit patterns are swept in the GPU
// tests); blocks that hold a NaN or an infinity take the integer encoder.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "rk_common.cuh"
#include "rk_internal.h"
#include "rk_rebase.cuh"

namespace rk {

int g_ring_stop = 0;   // set by rk_debug_set_ring_stop (tests only)
int g_rmsnorm_form = 0;   // set by rk_debug_set_rmsnorm_form (tests only)

template <int FMT> RK_DEVINL uint32_t ref_encode4(float a, float b, float c, float d) {
  return encode_rne<FMT>(a) | (encode_rne<FMT>(b) << 8) | (encode_rne<FMT>(c) << 16) | (encode_rne<FMT>(d) << 24);
}

// Sweeps fp32 bit patterns [first, first + count): counts inputs on which the hardware converter and the
// reference's integer encoder disagree (NaNs excluded: the kernels never hand one to the converter).
template <int FMT>
__global__ void verify_encoder_kernel(uint64_t first, uint64_t count, unsigned long long* mismatches, uint32_t* first_bad) {
  unsigned long long bad = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t bits = (uint32_t)(first + i);
    if ((bits & 0x7FFFFFFFu) > 0x7F800000u) continue;
    const float x = __uint_as_float(bits);
    const uint32_t hw = hw_encode4<FMT>(x, 0.0f, 0.0f, 0.0f) & 0xFFu;
    const uint32_t rf = encode_rne<FMT>(x);
    if (hw != rf) { if (bad == 0) atomicMin(first_bad, bits); ++bad; }
  }
  if (bad) atomicAdd(mismatches, bad);
}

// BF16IN: the input is bf16 (one 16-byte load per chunk, widened exactly to fp32) instead of fp32.
// LAYOUT: where a block's scale byte goes -- 0 row-major [rows][d/32]; 1 group-major [batch][d/32][S]; 2 the
// 512-byte scale-factor atoms [batch][ceil(S/128)][ceil(d/128)][512] the attention kernel copies into TMEM
// (S = rows per matrix of the batch, nbd = d/32; both unused for layout 0).
template <int FMT, bool BF16IN = false, int LAYOUT = 0>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const float4* __restrict__ x, int64_t nchunks,
                                                            uint2* __restrict__ codes, uint8_t* __restrict__ scales,
                                                            int64_t S = 0, int nbd = 0) {
  grid_dependency_wait();
  grid_dependents_launch();
  // chunk = 8 consecutive elements; 4 consecutive lanes = one 32-element block.
  // Warp-uniform loop bound: all 32 lanes run the shuffles even when the last
  // chunks of the array end inside this warp (nchunks is a multiple of 4, so a
  // 4-lane group is either wholly live or wholly idle).
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  // U chunks per trip, their loads issued together: the bf16 path loads half the bytes per chunk and gains 7 %
  // from two chunks in flight (measured); the fp32 path does not.
  constexpr int U = BF16IN ? 2 : 1;
  for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c0 - lane < nchunks; c0 += U * stride) {
    float4 a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t c = c0 + u * stride;
      a[u] = make_float4(0.f, 0.f, 0.f, 0.f); b[u] = a[u];
      if (c < nchunks) {
        if (BF16IN) {
          const float4 raw = __ldcs(x + c);                      // 8 bf16
          const uint32_t w[4] = {__float_as_uint(raw.x), __float_as_uint(raw.y), __float_as_uint(raw.z), __float_as_uint(raw.w)};
          a[u] = make_float4(__uint_as_float(w[0] << 16), __uint_as_float(w[0] & 0xFFFF0000u), __uint_as_float(w[1] << 16), __uint_as_float(w[1] & 0xFFFF0000u));
          b[u] = make_float4(__uint_as_float(w[2] << 16), __uint_as_float(w[2] & 0xFFFF0000u), __uint_as_float(w[3] << 16), __uint_as_float(w[3] & 0xFFFF0000u));
        } else {
          a[u] = __ldcs(x + 2 * c); b[u] = __ldcs(x + 2 * c + 1);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t c = c0 + u * stride;
      if (c - lane >= nchunks) break;                            // warp-uniform: the shuffles below need whole warps
      const bool live = c < nchunks;
      const float v[8] = {a[u].x, a[u].y, a[u].z, a[u].w, b[u].x, b[u].y, b[u].z, b[u].w};
      float amax = 0.0f, nonfinite = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        amax = fmaxf(amax, fabsf(v[j]));          // a NaN never wins, as in the reference's compare loop
        nonfinite = fmaf(v[j], 0.0f, nonfinite);  // stays 0 unless an element is NaN or +-inf
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      if (!live) continue;
      uint32_t scode = 0; float p2 = 1.0f;
      if (amax > 0.0f) block_scale<FMT>(amax, scode, p2);
      uint32_t w0, w1;
      if (nonfinite == 0.0f) {
        w0 = hw_encode4<FMT>(v[0] * p2, v[1] * p2, v[2] * p2, v[3] * p2);
        w1 = hw_encode4<FMT>(v[4] * p2, v[5] * p2, v[6] * p2, v[7] * p2);
      } else {
        w0 = ref_encode4<FMT>(v[0] * p2, v[1] * p2, v[2] * p2, v[3] * p2);
        w1 = ref_encode4<FMT>(v[4] * p2, v[5] * p2, v[6] * p2, v[7] * p2);
      }
      __stcs(codes + c, make_uint2(w0, w1));
      if ((c & 3) == 0) {
        if (LAYOUT == 0) {
          scales[c >> 2] = (uint8_t)scode;
        } else {
          const int64_t bi = c >> 2, row = bi / nbd, mat = row / S;
          const int blk = (int)(bi % nbd), r = (int)(row % S);
          if (LAYOUT == 1) {
            scales[(mat * nbd + blk) * S + r] = (uint8_t)scode;
          } else {
            const int64_t ntile = (S + 127) / 128, dch = (nbd + 3) / 4;
            scales[((mat * ntile + r / 128) * dch + blk / 4) * 512 + sf_atom_offset(r & 127, blk & 3)] = (uint8_t)scode;
          }
        }
      }
    }
  }
}

// 8 consecutive elements as loaded: 8 bf16 or 8 fp32.  PIECE = bytes per load instruction (16, or 4 for an unaligned base)
template <bool BF16IN> struct Raw8 { uint32_t w[BF16IN ? 4 : 8]; };
template <bool BF16IN, int PIECE> RK_DEVINL Raw8<BF16IN> load_raw8(const uint8_t* src) {
  constexpr int kWords = BF16IN ? 4 : 8;
  Raw8<BF16IN> r;
  if (PIECE == 16) {
#pragma unroll
    for (int i = 0; i < kWords / 4; ++i) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(src) + i);
      r.w[4 * i] = q.x; r.w[4 * i + 1] = q.y; r.w[4 * i + 2] = q.z; r.w[4 * i + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < kWords; ++i) r.w[i] = __ldg(reinterpret_cast<const uint32_t*>(src) + i);
  }
  return r;
}
// the same elements as fp32 (exact)
template <bool BF16IN> RK_DEVINL void widen8(const Raw8<BF16IN>& r, float (&v)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (BF16IN) v[j] = __uint_as_float((j & 1) ? (r.w[j / 2] & 0xFFFF0000u) : (r.w[j / 2] << 16));
    else v[j] = __uint_as_float(r.w[j]);
  }
}

// Pairs of fp32 in one 64-bit register.  (A product and a sum of pairs are contracted to one rounding, .rn or not: where both roundings count the products are scalar.)
RK_DEVINL uint64_t pair_u32(uint32_t a, uint32_t b) { uint64_t d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b)); return d; }
RK_DEVINL uint64_t pair_f32(float a, float b) { uint64_t d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
RK_DEVINL void unpair_u32(uint64_t p, uint32_t& a, uint32_t& b) { asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(p)); }
RK_DEVINL void unpair_f32(uint64_t p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
RK_DEVINL uint64_t mul_f32x2(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
RK_DEVINL uint64_t add_f32x2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
RK_DEVINL uint64_t fma_sq_f32x2(uint64_t v, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(v), "l"(c)); return d; }

// max(|a|, |b|, |c|), NaN if any of them is
RK_DEVINL float max3_abs_nan(float a, float b, float c) { float d; asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c)); return d; }
RK_DEVINL float max_nan(float a, float b) { float d; asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b)); return d; }

// One lane's 8 N elements of a 32-element block that 4 / N consecutive lanes share (they call together): the codes and the
// block's scale code.  Returns false where the block holds a NaN or an infinity (the maximum lets NaN through, so one
// comparison tells): its codes are then those of the COLD form, which takes the maximum without the NaNs, as the
// reference's compare loop does, and the integer encoder.  A caller runs the hot form over all it has and the cold one
// again only if some block asked for it, so that the hot loop carries no code that never runs.
// UNIT: no block scale (codes under 2^0, scale code 127).  PACKED: products two at a time, where issue slots are short (RMSNorm: 16384 x 4064 bf16
// 68.6 -> 67.2 us, 8192 x 4096 fp32 50.4 -> 49.6); scalar in the quantizer and RoPE, which HBM bounds: mul.f32x2 takes two cycles of the heavy FMA pipe, and packing its operands
// adds moves.
template <int FMT, bool UNIT, int N, bool COLD, bool PACKED = false> RK_DEVINL bool quantize_lanes(const float (&v)[N][8], int lane, uint2 (&w)[N], uint32_t& scode) {
  constexpr int kLanes = 4 / N;
  const uint32_t mask = (0xFu >> (4 - kLanes)) << (lane & (32 - kLanes));
  float m = 0.0f;
#pragma unroll
  for (int h = 0; h < N; ++h)
#pragma unroll
    for (int j = 0; j < 8; j += 2) m = COLD ? fmaxf(m, fmaxf(fabsf(v[h][j]), fabsf(v[h][j + 1]))) : max3_abs_nan(m, v[h][j], v[h][j + 1]);
#pragma unroll
  for (int s = 1; s < kLanes; s *= 2) {
    const float o = __shfl_xor_sync(mask, m, s);
    m = COLD ? fmaxf(m, o) : max_nan(m, o);
  }
  float p2 = 1.0f;
  scode = UNIT ? 127u : 0u;
  if (!UNIT && m > 0.0f) block_scale<FMT>(m, scode, p2);
#pragma unroll
  for (int h = 0; h < N; ++h) {
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      if (PACKED) unpair_f32(mul_f32x2(pair_f32(v[h][j], v[h][j + 1]), pair_f32(p2, p2)), s[j], s[j + 1]);
      else { s[j] = __fmul_rn(v[h][j], p2); s[j + 1] = __fmul_rn(v[h][j + 1], p2); }
    }
    w[h] = COLD ? make_uint2(ref_encode4<FMT>(s[0], s[1], s[2], s[3]), ref_encode4<FMT>(s[4], s[5], s[6], s[7]))
                : make_uint2(hw_encode4<FMT>(s[0], s[1], s[2], s[3]), hw_encode4<FMT>(s[4], s[5], s[6], s[7]));
  }
  return m < __int_as_float(0x7f800000);
}

// RoPE fused with the block quantizer, so that rotated Q / K never exist in HBM as fp32: rotate-half form with
// half-width caches (lib/golden/golden.py:229-236): out[:half] = c0 cos - c1 sin, out[half:] = c1 cos + c0 sin,
// every product and sum rounded on its own (no fused multiply-add, as numpy float32 does), then the lib/golden block
// rule along d.  chunk = 8 consecutive elements of the first half and their 8 partners of the second half; 4 lanes
// = one 32-element block in each half.  Row r uses cache row pos[r], or pos0 + r % seq_len when pos is null.
// U rows of the same position (heads, sequences: rows seq_len apart) per thread share what it reads of the caches, which
// otherwise cost as many bytes from L2 as the rows do from HBM: 33.5 M elements 31 us with U = 1, 29 with 2.  U = 1 with a
// position list.
template <int FMT, int U, bool COLD>
RK_DEVINL bool rope_rows(const float* __restrict__ x, int64_t rows, int d, const int32_t* __restrict__ pos, int seq_len, int pos0,
                         const float* __restrict__ cos_h, const float* __restrict__ sin_h, uint8_t* __restrict__ codes,
                         uint8_t* __restrict__ scales) {
  const int half = d / 2, cpr = half / 8;                     // chunks per row (a multiple of 4)
  const int64_t period = U > 1 ? seq_len : rows;              // rows before the position repeats
  const int64_t copies = rows / period, per_copy = period * cpr, total = (copies + U - 1) / U * per_copy;
  bool finite = true;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < total; c += (int64_t)gridDim.x * blockDim.x) {
    int64_t bg, r0;
    int i0;
    if (total < (int64_t)1 << 31) {                           // 32-bit divisions whenever the index fits
      const uint32_t q = (uint32_t)c / (uint32_t)cpr;
      i0 = (int)((uint32_t)c - q * (uint32_t)cpr) * 8;
      const uint32_t g = q / (uint32_t)period;
      r0 = q - g * (uint32_t)period;
      bg = g;
    } else {
      const int64_t q = c / cpr;
      i0 = (int)(c - q * cpr) * 8;
      bg = q / period;
      r0 = q - bg * period;
    }
    const int64_t first = bg * U * period + r0;
    const int n = (int)min((int64_t)U, copies - bg * U);
    float4 a[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u < n) {
        const float4* xr = reinterpret_cast<const float4*>(x + (first + u * period) * d + i0);
        a[u][0] = __ldcs(xr); a[u][1] = __ldcs(xr + 1);
        a[u][2] = __ldcs(xr + half / 4); a[u][3] = __ldcs(xr + half / 4 + 1);
      }
    }
    const int64_t at = pos ? (int64_t)pos[first] : (int64_t)pos0 + (U > 1 ? r0 : r0 % seq_len);
    const float4* cp = reinterpret_cast<const float4*>(cos_h + at * half + i0);
    const float4* sp = reinterpret_cast<const float4*>(sin_h + at * half + i0);
    const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
    const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;                                      // the four lanes of a block agree
      const float lo[8] = {a[u][0].x, a[u][0].y, a[u][0].z, a[u][0].w, a[u][1].x, a[u][1].y, a[u][1].z, a[u][1].w};
      const float hi[8] = {a[u][2].x, a[u][2].y, a[u][2].z, a[u][2].w, a[u][3].x, a[u][3].y, a[u][3].z, a[u][3].w};
      float o0[1][8], o1[1][8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        o0[0][j] = __fsub_rn(__fmul_rn(lo[j], cs[j]), __fmul_rn(hi[j], sn[j]));
        o1[0][j] = __fadd_rn(__fmul_rn(hi[j], cs[j]), __fmul_rn(lo[j], sn[j]));
      }
      uint2 w0[1], w1[1];
      uint32_t sc0, sc1;
      finite &= quantize_lanes<FMT, false, 1, COLD>(o0, lane, w0, sc0);
      finite &= quantize_lanes<FMT, false, 1, COLD>(o1, lane, w1, sc1);
      const int64_t r = first + u * period;
      __stcs(reinterpret_cast<uint2*>(codes + r * d + i0), w0[0]);
      __stcs(reinterpret_cast<uint2*>(codes + r * d + half + i0), w1[0]);
      if ((lane & 3) == 0) {
        scales[r * (d / 32) + i0 / 32] = (uint8_t)sc0;
        scales[r * (d / 32) + (half + i0) / 32] = (uint8_t)sc1;
      }
    }
  }
  return finite;
}
template <int FMT, int U>
__global__ void __launch_bounds__(128) rope_quantize_rows_kernel(const float* __restrict__ x, int64_t rows, int d,
                                                                 const int32_t* __restrict__ pos, int seq_len, int pos0,
                                                                 const float* __restrict__ cos_h, const float* __restrict__ sin_h,
                                                                 uint8_t* __restrict__ codes, uint8_t* __restrict__ scales) {
  grid_dependency_wait();
  grid_dependents_launch();
  const bool finite = rope_rows<FMT, U, false>(x, rows, d, pos, seq_len, pos0, cos_h, sin_h, codes, scales);
  if (__syncthreads_or(!finite)) rope_rows<FMT, U, true>(x, rows, d, pos, seq_len, pos0, cos_h, sin_h, codes, scales);      // the same rows
}

// The same for large inputs with several rows per position: a CTA has a range of positions, kTileBytes of one head's rows, keeps what it needs of the caches in
// registers and walks every gridDim.y-th head, the next one's rows on their way by a bulk copy.  HBM bound (134 MB in and 35 MB out, which stay in L2 here:
// 21 us as the plain quantizer does it) once enough warps are there for a row's instructions: 33.5 M elements 30.7 us with two rows per thread in registers (117
// of them, 16 warps per SM), 31.2 with the next two rows loaded ahead (96, 20 warps), 28.4 by bulk copies four deep (24 warps), 27.8 now (64 registers, 32
// warps), 32.5 with 40 warps of 48 registers.
namespace ropec {
constexpr int kThreads = 128, kCtasPerSm = 8, kStages = 2, kTileBytes = kThreads * 64;      // a thread has 8 elements of either half of a row
}  // namespace ropec
struct RopeRing { uint8_t* data; uint64_t* full; uint32_t loads; };      // loads: so far
template <int FMT, bool COLD, bool STOPS>
RK_DEVINL bool rope_copies(const float* __restrict__ x, int copies, int d, int seq_len, int pos0, const float* __restrict__ cos_h,
                           const float* __restrict__ sin_h, uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, RopeRing& ring, int* status) {
  using namespace ropec;
  const int half = d / 2, cpr = half / 8, lane = threadIdx.x & 31, groups = gridDim.y;
  const int per_tile = kTileBytes / (d * 4), p0 = blockIdx.x * per_tile, n_rows = min(per_tile, seq_len - p0);
  const int row = threadIdx.x / cpr, i0 = (threadIdx.x - row * cpr) * 8;
  const bool live = row < n_rows;                             // (the four lanes of a block agree)
  const uint32_t bytes = (uint32_t)n_rows * d * 4;
  auto load = [&](int u, uint32_t n) {                        // rows of copy u, the n-th load
    uint64_t* bar = &ring.full[n % kStages];
    mbar_arrive_expect_tx(bar, bytes);
    bulk_load_1d(ring.data + (n % kStages) * kTileBytes, x + ((int64_t)u * seq_len + p0) * d, bytes, bar);
  };
  auto wait = [&](uint32_t n) -> bool {                       // bounded by 2^19 polls
#pragma unroll 1
    for (int it = 0; it < 1 << 19; ++it)
      if (mbar_try_wait<2000>(&ring.full[n % kStages], (n / kStages) & 1)) return true;
    return false;
  };
  const int first = blockIdx.y, mine = (copies - first + groups - 1) / groups;
  if (threadIdx.x == 0)
    for (int k = 0; k < min(mine, kStages); ++k) load(first + k * groups, ring.loads + k);
  float cs[8], sn[8];
  if (live) {
    const int64_t at = ((int64_t)pos0 + p0 + row) * half + i0;
    const float4* cp = reinterpret_cast<const float4*>(cos_h + at);
    const float4* sp = reinterpret_cast<const float4*>(sin_h + at);
    const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
    cs[0] = c0.x; cs[1] = c0.y; cs[2] = c0.z; cs[3] = c0.w; cs[4] = c1.x; cs[5] = c1.y; cs[6] = c1.z; cs[7] = c1.w;
    sn[0] = s0.x; sn[1] = s0.y; sn[2] = s0.z; sn[3] = s0.w; sn[4] = s1.x; sn[5] = s1.y; sn[6] = s1.z; sn[7] = s1.w;
  }
  bool finite = true;
  for (int k = 0; k < mine; ++k) {
    const uint32_t n = ring.loads + k;
    const bool there = wait(n) && !(STOPS && k == 1);          // (test hook: as if the wait had run out)
    const float4* src = reinterpret_cast<const float4*>(ring.data + (n % kStages) * kTileBytes + (live ? row : 0) * d * 4 + i0 * 4);      // (a branch around the loads: 8.98 us instead of 8.3 for 8.4 M elements)
    const float4 a0 = src[0], a1 = src[1], a2 = src[half / 4], a3 = src[half / 4 + 1];
    if (__syncthreads_or(!there)) {                           // (and read by all: the place is free)
      if (threadIdx.x == 0) {
        atomicCAS(status, 0, 601);
        for (int i = k; i < min(mine, k + kStages); ++i) wait(ring.loads + i);      // what is under way
      }
      return true;
    }
    if (threadIdx.x == 0 && k + kStages < mine) load(first + (k + kStages) * groups, n + kStages);
    if (live) {
      const float lo[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float hi[8] = {a2.x, a2.y, a2.z, a2.w, a3.x, a3.y, a3.z, a3.w};
      float o0[1][8], o1[1][8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        o0[0][j] = __fsub_rn(__fmul_rn(lo[j], cs[j]), __fmul_rn(hi[j], sn[j]));
        o1[0][j] = __fadd_rn(__fmul_rn(hi[j], cs[j]), __fmul_rn(lo[j], sn[j]));
      }
      uint2 w0[1], w1[1];
      uint32_t sc0, sc1;
      finite &= quantize_lanes<FMT, false, 1, COLD>(o0, lane, w0, sc0);
      finite &= quantize_lanes<FMT, false, 1, COLD>(o1, lane, w1, sc1);
      const int64_t r = (int64_t)(first + k * groups) * seq_len + p0 + row;
      __stcs(reinterpret_cast<uint2*>(codes + r * d + i0), w0[0]);
      __stcs(reinterpret_cast<uint2*>(codes + r * d + half + i0), w1[0]);
      if ((lane & 3) == 0) {
        scales[r * (d / 32) + i0 / 32] = (uint8_t)sc0;
        scales[r * (d / 32) + (half + i0) / 32] = (uint8_t)sc1;
      }
    }
  }
  ring.loads += mine;
  return finite;
}
template <int FMT, bool STOPS>
__global__ void __launch_bounds__(ropec::kThreads, ropec::kCtasPerSm)
rope_quantize_copies_kernel(const float* __restrict__ x, int copies, int d, int seq_len, int pos0, const float* __restrict__ cos_h, const float* __restrict__ sin_h,
                            uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, int* status) {
  __shared__ __align__(128) uint8_t rope_data[ropec::kStages * ropec::kTileBytes];
  __shared__ uint64_t rope_full[ropec::kStages];
  if (threadIdx.x < ropec::kStages) mbar_init(&rope_full[threadIdx.x], 1);
  fence_barrier_init();
  __syncthreads();
  grid_dependency_wait();
  grid_dependents_launch();
  RopeRing ring = {rope_data, rope_full, 0};
  const bool finite = rope_copies<FMT, false, STOPS>(x, copies, d, seq_len, pos0, cos_h, sin_h, codes, scales, ring, status);
  if (__syncthreads_or(!finite)) rope_copies<FMT, true, STOPS>(x, copies, d, seq_len, pos0, cos_h, sin_h, codes, scales, ring, status);      // the same rows
}

// RMSNorm fused with the block quantizer: the prologue of the QKV projection (kernels/rmsnorm_qkv_fused), so that the
// normalized activation never exists in HBM as fp32.  Bit-exact with the reference's fp32 path
// (lib/golden/golden.py:203-216): the sum of squares runs in index order with every product and sum rounded on its
// own, mean = ss / K, rms = 1 / sqrt(mean + eps) (correctly rounded square root and division), y = (x * rms) * gamma.
// UNIT: no block scale (code = E4M3(y) under 2^0, every scale byte 0x7F), the reference kernel's own choice
// (kernels/rmsnorm_qkv_fused/gen_data.py:33-41: the prologue owns the row scaling).
//
// The index-order sum is a chain of K dependent additions per row, 4.3 cycles each: 9 us for K = 4096, about what the
// input takes to arrive from HBM.  So all chains of the machine run at once -- a CTA owns up to 16 rows, one lane of one
// warp each -- and that warp does nothing but 16-byte shared-memory reads and additions (5.1 cycles a step alone on its
// scheduler, 6.7 beside the other CTAs; with the squares in its own instruction stream 6.4 and 9).  Four other warps load
// the rows two chunks of 256 elements ahead in registers and leave the squares in one of two buffers whose row pitch (1040
// bytes) gives eight lanes reading 16 bytes of their own rows eight different bank groups.  When the chains are done all
// warps normalize and quantize; the input then comes from L2 (DRAM reads it once).  Over the whole kernel 53 % of the issue
// slots and 22 % of DRAM's rate are used: the two phases of a CTA run one after the other, and neither fills the machine.
// 8192 x 4096 bf16: 1362 us with one warp per 32 rows doing both passes from 4-byte shared-memory reads, 36.5 us this way, 31.8 by bulk copies (below).
namespace rms {
constexpr int kThreads = 256, kHelpers = 4, kCtasPerSm = 4;
constexpr int kChunk = 256, kPitch = kChunk * 4 + 16, kBufs = 2;        // elements per chunk, bytes of a row of squares
constexpr int kHalf = kChunk / 8;                                       // float4s of a row: first halves of the lanes' eight, then second
constexpr int kMaxRows = 16;
constexpr int kRowsPerHelper = (kMaxRows + kHelpers - 1) / kHelpers;
constexpr int kFull = 1, kEmpty = kFull + kBufs;                        // named barriers
}  // namespace rms
// barrier ID or ID + 1 (constants: a register would make the kernel claim all sixteen)
template <int ID> RK_DEVINL void named_sync(int which) {
  if (which) asm volatile("bar.sync %0, %1;" ::"n"(ID + 1), "n"((1 + rms::kHelpers) * 32) : "memory");
  else asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"((1 + rms::kHelpers) * 32) : "memory");
}
template <int ID> RK_DEVINL void named_arrive(int which) {
  if (which) asm volatile("bar.arrive %0, %1;" ::"n"(ID + 1), "n"((1 + rms::kHelpers) * 32) : "memory");
  else asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"((1 + rms::kHelpers) * 32) : "memory");
}

constexpr int kPieceShared = 0;                                         // PIECE of rows that lie in shared memory
template <bool BF16IN, int PIECE>
RK_DEVINL void load_pair(Raw8<BF16IN> (&r)[2], const uint8_t* src, bool a32) {
  if (PIECE == kPieceShared) {
    constexpr int kQuads = BF16IN ? 1 : 2;
#pragma unroll
    for (int i = 0; i < 2 * kQuads; ++i) {
      const uint4 q = reinterpret_cast<const uint4*>(src)[i];
      uint32_t* w = r[i / kQuads].w + 4 * (i % kQuads);
      w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
    }
  } else if (BF16IN && PIECE == 16 && a32) {
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0].w[0]), "=r"(r[0].w[1]), "=r"(r[0].w[2]), "=r"(r[0].w[3]), "=r"(r[1].w[0]), "=r"(r[1].w[1]), "=r"(r[1].w[2]), "=r"(r[1].w[3]) : "l"(src));
  } else { r[0] = load_raw8<BF16IN, PIECE>(src); r[1] = load_raw8<BF16IN, PIECE>(src + 8 * (BF16IN ? 2 : 4)); }
}
// The second phase of the RMSNorm kernels: y = (x rms) gamma of the CTA's rows, quantized.  rms_smem: shared memory to put the scale bytes together in,
// room bytes of it for every row.
template <int FMT, bool BF16IN, bool UNIT, int PIECE, int kThreads>
RK_DEVINL void rmsnorm_rows(const uint8_t* __restrict__ xr, int64_t row0, int n_rows, int K, const float* __restrict__ gamma, const float* rms_row,
                            uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, uint8_t* rms_smem, int room) {
  constexpr int kElem = BF16IN ? 2 : 4, kWarps = kThreads / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row_bytes = (int64_t)K * kElem;
  // ---- normalize and quantize: a warp keeps 512 columns (16 per lane, 2 lanes per block; gamma in registers) and walks
  // the rows, the load of one more row in flight; with fewer column units than warps several warps share one ------------
  // (Scale bytes meet in shared memory first: a byte store per 32 elements cost a fifth of this phase.)
  const bool stage_scales = K / 32 <= room;                   // they fit where the squares were
  const bool a32 = (reinterpret_cast<uintptr_t>(xr) & 31) == 0;
  const int per_row = (K + 511) / 512, parts = max(1, kWarps / per_row);
  const int part = warp / per_row;
  auto quantize_rows = [&](auto cold_tag) -> bool {
    constexpr bool COLD = decltype(cold_tag)::value;
    bool finite = true;
    if (part >= parts) return finite;
    for (int u = warp - part * per_row; u < per_row; u += kWarps) {
      const int col = u * 512 + lane * 16;
      if (col >= K) continue;                                           // whole 2-lane groups: K % 32 == 0
      const int64_t src_step = parts * row_bytes, dst_step = (int64_t)parts * K;
      const int sc_step = parts * (K / 32);
      const uint8_t* src = xr + part * row_bytes + (int64_t)col * kElem;
      uint8_t* dst = codes + (row0 + part) * K + col;
      uint8_t* sdst = (stage_scales ? rms_smem : scales + row0 * (K / 32)) + part * (K / 32) + col / 32;
      float g[2][8];
      widen8<false>(load_raw8<false, PIECE>(reinterpret_cast<const uint8_t*>(gamma + col)), g[0]);
      widen8<false>(load_raw8<false, PIECE>(reinterpret_cast<const uint8_t*>(gamma + col + 8)), g[1]);
      Raw8<BF16IN> raw[2];
      if (part < n_rows) load_pair<BF16IN, PIECE>(raw, src, a32);
      src += src_step;
#pragma unroll 1
      for (int r = part; r < n_rows; r += parts) {
        const float rms = rms_row[r];
        float v[2][8];
        widen8<BF16IN>(raw[0], v[0]);
        widen8<BF16IN>(raw[1], v[1]);
        if (r + parts < n_rows) load_pair<BF16IN, PIECE>(raw, src, a32);
        src += src_step;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 8; j += 2)
            unpair_f32(mul_f32x2(mul_f32x2(pair_f32(v[h][j], v[h][j + 1]), pair_f32(rms, rms)), pair_f32(g[h][j], g[h][j + 1])), v[h][j], v[h][j + 1]);
        uint32_t scode;
        uint2 w[2];
        finite &= quantize_lanes<FMT, UNIT, 2, COLD, true>(v, lane, w, scode);
        __stcs(reinterpret_cast<uint4*>(dst), make_uint4(w[0].x, w[0].y, w[1].x, w[1].y));
        if ((lane & 1) == 0) *sdst = (uint8_t)scode;
        dst += dst_step;
        sdst += sc_step;
      }
    }
    return finite;
  };
  if (__syncthreads_or(!quantize_rows(std::false_type{}))) quantize_rows(std::true_type{});
  if (stage_scales) {
    __syncthreads();
    const int n = n_rows * (K / 32);                                    // contiguous in memory, as the CTA's rows are
    uint8_t* out = scales + row0 * (K / 32);
    if ((reinterpret_cast<uintptr_t>(out) & 3) == 0 && (n & 3) == 0) {
      for (int i = threadIdx.x; i < n / 4; i += kThreads) reinterpret_cast<uint32_t*>(out)[i] = reinterpret_cast<const uint32_t*>(rms_smem)[i];
    } else {
      for (int i = threadIdx.x; i < n; i += kThreads) out[i] = rms_smem[i];
    }
  }
}

// PIECE: bytes of one global load: 16, or 4 where x or gamma is not 16-byte aligned.
template <int FMT, bool BF16IN, bool UNIT, int PIECE>
__global__ void __launch_bounds__(rms::kThreads, rms::kCtasPerSm)
rmsnorm_quantize_kernel(const uint8_t* __restrict__ x, int64_t rows, int K, int rows_per_cta, const float* __restrict__ gamma,
                        float eps, uint8_t* __restrict__ codes, uint8_t* __restrict__ scales) {
  grid_dependency_wait();
  grid_dependents_launch();
  using namespace rms;
  extern __shared__ __align__(16) uint8_t rms_smem[];                   // [kBufs][n_rows][kPitch] squares
  __shared__ float rms_row[kMaxRows];
  constexpr int kElem = BF16IN ? 2 : 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Schedulers: the chains run on the first two, the squares on the other two (a burst of squares beside a chain takes
  // its issue slots).  Blocks go to the SMs in rounds of gridDim / kCtasPerSm: alternate rounds take warp 0 and warp 1.
  const int chain_warp = (int)(blockIdx.x / ((gridDim.x + kCtasPerSm - 1) / kCtasPerSm)) & 1;
  const int helper = (warp & 2) ? (warp & 1) + (warp >> 2) * 2 : -1;       // warps 2, 3, 6, 7
  const int64_t row0 = (int64_t)blockIdx.x * rows_per_cta;
  const int n_rows = (int)min((int64_t)rows_per_cta, rows - row0);
  const int64_t row_bytes = (int64_t)K * kElem;
  const uint8_t* xr = x + row0 * row_bytes;
  const int n_chunks = (K + kChunk - 1) / kChunk;
  const int buf_bytes = n_rows * kPitch;

  if (warp == chain_warp) {
    // ---- the chains ---------------------------------------------------------------------------------------------
    float ss = 0.0f;
    for (int c = 0; c < n_chunks; ++c) {
      named_sync<kFull>(c & 1);
      if (lane < n_rows) {
        const float4* src = reinterpret_cast<const float4*>(rms_smem + (c & 1) * buf_bytes + lane * kPitch);
        const int n4 = min(kChunk, K - c * kChunk) / 4;                 // a multiple of 8
        float4 s[3][4];
        auto fetch = [&](int i, float4 (&d)[4]) {
#pragma unroll
          for (int q = 0; q < 4; ++q) d[q] = src[(q & 1) * kHalf + i / 2 + q / 2];
        };
        auto chain = [&](const float4 (&d)[4]) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            ss = __fadd_rn(ss, d[q].x); ss = __fadd_rn(ss, d[q].y);
            ss = __fadd_rn(ss, d[q].z); ss = __fadd_rn(ss, d[q].w);
          }
        };
        fetch(0, s[0]);                                                 // two batches of sixteen additions ahead
        fetch(4, s[1]);
        int i = 0;
        for (; i + 20 <= n4; i += 12) {
          fetch(i + 8, s[2]); chain(s[0]);
          fetch(i + 12, s[0]); chain(s[1]);
          fetch(i + 16, s[1]); chain(s[2]);
        }
        for (; i < n4; i += 4) {
          chain(s[0]);
#pragma unroll
          for (int q = 0; q < 4; ++q) s[0][q] = s[1][q];
          if (i + 8 < n4) fetch(i + 8, s[1]);
        }
      }
      __syncwarp();
      if (c + kBufs < n_chunks) named_arrive<kEmpty>(c & 1);
    }
    if (lane < n_rows) rms_row[lane] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  } else if (helper >= 0) {
    // ---- squares: rows helper, helper + 4, ... of every chunk, two chunks ahead in registers (one for fp32 input) -------
    constexpr int kAhead = BF16IN ? 2 : 1;
    Raw8<BF16IN> raw[kAhead][kRowsPerHelper];
    const int n_mine = (n_rows - helper + kHelpers - 1) / kHelpers;     // rows of this warp
    const int64_t row_step = kHelpers * row_bytes;
    const uint8_t* src = xr + helper * row_bytes + lane * 8 * kElem;    // advances by a chunk with every fetch
    float4* const dst0 = reinterpret_cast<float4*>(rms_smem + helper * kPitch) + lane;
    auto fetch = [&](int c, Raw8<BF16IN> (&d)[kRowsPerHelper]) {
      if (c * kChunk + lane * 8 < K) {
        const uint8_t* q = src;
#pragma unroll
        for (int k = 0; k < kRowsPerHelper; ++k) {
          if (k < n_mine) d[k] = load_raw8<BF16IN, PIECE>(q);
          q += row_step;
        }
      }
      src += kChunk * kElem;
    };
    auto square = [&](int c, const Raw8<BF16IN> (&d)[kRowsPerHelper]) {
      if (c >= kBufs) named_sync<kEmpty>(c & 1);
      float4* dst = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(dst0) + (c & 1) * buf_bytes);
      if (c * kChunk + lane * 8 < K) {
#pragma unroll
        for (int k = 0; k < kRowsPerHelper; ++k) {
          if (k < n_mine) {
            float v[8];
            widen8<BF16IN>(d[k], v);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(v[j], v[j]);
            dst[k * (kHelpers * kPitch / 16)] = make_float4(v[0], v[1], v[2], v[3]);
            dst[k * (kHelpers * kPitch / 16) + kHalf] = make_float4(v[4], v[5], v[6], v[7]);
          }
        }
      }
      named_arrive<kFull>(c & 1);
    };
#pragma unroll
    for (int a = 0; a < kAhead; ++a) fetch(a, raw[a]);
    for (int c = 0; c < n_chunks; c += kAhead) {
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        if (c + a < n_chunks) {
          square(c + a, raw[a]);
          fetch(c + a + kAhead, raw[a]);
        }
      }
    }
  }
  __syncthreads();

  rmsnorm_rows<FMT, BF16IN, UNIT, PIECE, kThreads>(xr, row0, n_rows, K, gamma, rms_row, codes, scales, rms_smem, kBufs * kPitch);
}

// The same for bf16 rows, which come by bulk copies, a warp's lanes each asking for one row's next 1024 bytes; the chain warp, up to 32 rows of it in lanes,
// squares what it reads itself, and no other warp has anything to do with the rows until the chains are done.  A chain step takes 5.1 cycles as a fused
// multiply-add (4.3 the addition alone), 6 as a product and a sum in one instruction stream, against 6.1 with one row and 10 with 8192 of them staged through
// other warps' registers and shared memory as squares, two barriers per 256 elements.  The square of a bf16 is exact in fp32, so fusing changes nothing, unless
// it is below 2^-133; where the first element of every row is 2^-50 or more, such a square is less than half a step of any sum and adds nothing
// either way.  Other rows (that begin with a zero, say) keep products and sums.  16384 x 4064: 67.2 -> 66.1 us, 16384 x 2048 36.5 -> 35.8.
// 8192 x 4096: 36.5 -> 31.8 us (inputs that change from call to call 34.5, fused 33.7), about half of it the chains, half the quantization from L2 (67 MB in, 35 MB out). The
// pieces that are still in shared memory read from there: no change.  The quantization with one 32-byte load per
// lane and row, one row ahead: two rows ahead 37.2, 16-byte loads two rows ahead 34.0.  Four CTAs of 256 threads 38.8, one of 1024 49.8.
namespace rmb {
constexpr int kThreads = 512, kCtasPerSm = 2, kMaxRows = 32, kStages = 3, kPieceBytes = 1024, kPitch = kPieceBytes + 16;      // pitch: eight lanes, eight bank groups
}  // namespace rmb
template <int FMT, bool UNIT, bool STOPS>
__global__ void __launch_bounds__(rmb::kThreads, rmb::kCtasPerSm)
rmsnorm_quantize_bulk_kernel(const uint8_t* __restrict__ x, int64_t rows, int K, int rows_per_cta, const float* __restrict__ gamma,
                             float eps, uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, int* status, int stop) {
  using namespace rmb;
  extern __shared__ __align__(16) uint8_t rmb_smem[];                   // [kStages][n_rows][kPitch]
  __shared__ float rms_row[kMaxRows];
  __shared__ uint64_t full[kStages], empty[kStages];
  constexpr int kElem = 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kStages) { mbar_init(&full[threadIdx.x], 1); mbar_init(&empty[threadIdx.x], 1); }
  fence_barrier_init();
  __syncthreads();
  grid_dependency_wait();
  grid_dependents_launch();
  const int64_t row0 = (int64_t)blockIdx.x * rows_per_cta;
  const int n_rows = (int)min((int64_t)rows_per_cta, rows - row0);
  const int64_t row_bytes = (int64_t)K * kElem;
  const uint8_t* xr = x + row0 * row_bytes;
  const int n_pieces = (int)((row_bytes + kPieceBytes - 1) / kPieceBytes), stage_bytes = n_rows * kPitch;
  // the chains of the CTAs of an SM on schedulers of their own: blocks go to the SMs in rounds of gridDim / kCtasPerSm
  const int chain_warp = (int)(blockIdx.x / ((gridDim.x + kCtasPerSm - 1) / kCtasPerSm)) % kCtasPerSm;
  bool ok = true;
  int issued = 0;                                                       // pieces the producer has asked for
  auto wait = [&](uint64_t* bar, int use) -> bool {                     // bounded by 2^19 polls, about two seconds (a look at a flag of the other role's: 1-2 % of a call)
#pragma unroll 1
    for (int it = 0; it < 1 << 19; ++it)
      if (mbar_try_wait<2000>(bar, use & 1)) return true;
    return false;
  };
  auto stops = [&](int role, int c) { return STOPS && stop == role && c == kStages + 1; };      // test hook: the role acts as if its wait had run out
  if (warp == chain_warp) {
    float ss = 0.0f;
    // elements 8 i to 8 (i + n16) of a piece, as products and sums or as fused multiply-adds
    auto add_piece = [&](const uint4* src, int n16, auto fused_tag) {
      constexpr bool kFused = decltype(fused_tag)::value;
      constexpr int kSq = 16 / kElem;                                   // elements of 16 bytes
      auto widen = [&](const uint4& q, float (&d)[kSq]) {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xFFFF0000u);
          d[2 * j] = kFused ? lo : __fmul_rn(lo, lo);
          d[2 * j + 1] = kFused ? hi : __fmul_rn(hi, hi);
        }
      };
      auto chain = [&](const float (&d)[kSq]) {
#pragma unroll
        for (int j = 0; j < kSq; ++j) ss = kFused ? __fmaf_rn(d[j], d[j], ss) : __fadd_rn(ss, d[j]);
      };
      uint4 q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = src[k];
      float d[2][kSq];
      widen(q[0], d[0]);
#pragma unroll 1
      for (int i = 0; i < n16; i += 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {                                   // elements a piece of 16 bytes ahead, loads four
          if (i + k + 4 < n16) q[k] = src[i + k + 4];
          widen(q[(k + 1) & 3], d[(k + 1) & 1]);
          chain(d[k & 1]);
        }
      }
    };
    bool fused = false;
    for (int c = 0; c < n_pieces && ok; ++c) {
      const int st = c % kStages;
      ok = __all_sync(0xffffffffu, !stops(1, c) && wait(&full[st], c / kStages));
      if (!ok) break;
      const uint4* src = reinterpret_cast<const uint4*>(rmb_smem + st * stage_bytes + lane * kPitch);
      if (c == 0) fused = __all_sync(0xffffffffu, lane >= n_rows || (src[0].x & 0x7FFFu) >= (127u - 50u) << 7);
      if (lane < n_rows) {
        const int n16 = (int)min((int64_t)kPieceBytes, row_bytes - (int64_t)c * kPieceBytes) / 16;      // a multiple of 4
        if (fused) add_piece(src, n16, std::true_type{}); else add_piece(src, n16, std::false_type{});
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[st]);
    }
    if (lane < n_rows) rms_row[lane] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  } else if (warp == kThreads / 32 - 1) {
    for (int c = 0; c < n_pieces && ok; ++c) {
      const int st = c % kStages;
      if (c >= kStages) ok = __all_sync(0xffffffffu, !stops(2, c) && wait(&empty[st], c / kStages - 1));
      if (!ok) break;
      const uint32_t bytes = (uint32_t)min((int64_t)kPieceBytes, row_bytes - (int64_t)c * kPieceBytes);
      if (lane == 0) mbar_arrive_expect_tx(&full[st], bytes * n_rows);
      __syncwarp();
      if (lane < n_rows) bulk_load_1d(rmb_smem + st * stage_bytes + lane * kPitch, xr + lane * row_bytes + (int64_t)c * kPieceBytes, bytes, &full[st]);
      ++issued;
    }
  }
  if (__syncthreads_or(!ok)) {
    // the copies under way, whichever role gave up, before shared memory goes to another CTA
    for (int c = max(0, issued - kStages); c < issued; ++c) wait(&full[c % kStages], c / kStages);
    if (threadIdx.x == 0) atomicCAS(status, 0, 602);                   // an RMSNorm call's copies, in this kernel and the one below
    return;
  }
  rmsnorm_rows<FMT, true, UNIT, 16, kThreads>(xr, row0, n_rows, K, gamma, rms_row, codes, scales, rmb_smem, kStages * kPitch);
}

// The same where every row is on the chip at once and few of them share an SM: the chain of a row is cut into segments that lanes walk side by side.
// As long as an index-order sum stays in one binade [2^e, 2^(e+1)) with steps of u between its fp32 values, adding x >= 0 with round to nearest even
// commutes with a shift of the sum by a multiple of 2u: what a segment adds depends only on whether the sum before it is an even or an odd multiple of u.
// So each segment is added up twice, from 2^e and from 2^e + u, two segments of a lane side by side, and its result is the pair of gains in steps of u; runs
// of segments of one binade compose to such a pair.  e comes from sums in another order, which are off by little: a segment whose guess may be wrong, or in
// which the binade ends, is marked, as are those below 2^-87 (for bf16 the chains are fused multiply-adds: a square is exact in fp32, or below 2^-133 and
// then no part of a sum of 2^-87 and more).  In the end one lane per row goes over the runs with the sum itself, asks of each run that the sum starts and ends in the
// binade the gain was taken in -- sums only grow, so it has then been there all along -- and adds what is marked, or fails the question, in order as it lies.
// Any input gives the bits of the index-order sum; a wrong guess costs time.  (N(0,1): a segment per doubling of the sum, 7 or 8 of the 103 of 4096 columns.)
// Rows that are marked throughout -- sums below 2^-87, an infinity or a NaN -- are added up by that lane alone: marked segments side by side are one run, four
// pieces of 16 bytes at a time, so that the addition's latency is what counts.  One row of 4096 bf16 of 2^-52 N(0,1) 17.6 us (the chain as it lies in the ring 15.6, a run per segment
// 40.7), fp32 19.7 (17.2, 76.3), 300 rows of 12288 bf16 49.6 (45.7, 155.6), 1200 of 4096 24.0 (19.5, 47.6); N(0,1) gains by it too (300 rows of 4096 fp32 11.0 -> 9.8, one 9.0 -> 7.7).
//
// One row of 4096 bf16: 15.7 -> 7.2 us, 12288 columns 42.1 -> 10.0; 300 rows of 4096 17.5 -> 8.9, 1500 rows 19.8 -> 13.9; fp32, one row of 4096 17.3 -> 7.4.  With more rows on an SM than its shared
// memory holds the rounds of CTAs follow one another with little overlap, and the ring above, whose chains all run at once, is faster (4500 rows 25.3, so 33.8).
// The quantization reads the rows where they are; products two at a time (88 instead of 112 instructions per 16 elements and lane).
namespace rms_seg {
constexpr int kThreads = 256, kWarps = kThreads / 32, kCtasPerSm = 3, kMaxRows = 8;
constexpr int kSmem = 227 * 1024, kStatic = 1024, kReserved = 1024;     // of an SM; of a CTA beside its dynamic part, ours and the system's
constexpr uint32_t kMarked = 0x3FF;                                     // in the place of an exponent
constexpr int kLongest = 72;                                            // elements of a segment, before they are rounded up to whole pieces (24 to 72 bf16, 20 to 76 fp32 then)

// How a call is laid out: rows per CTA, warps that share a row's segments, segment in elements, bytes from row to row in shared memory.
struct Shape { int rows, warps, seg, pitch; int64_t smem, grid; };
// Segments are an odd number of 16-byte pieces, so that eight lanes reading 16 bytes of their own find eight bank groups.
static Shape shape(int64_t n, int K, bool bf16, int rows) {
  const int elem = bf16 ? 2 : 4, piece = 16 / elem, least = rows == 1 && !bf16 ? 24 : 40;      // elements: a row goes to more warps while their segments are longer than these
  Shape f;
  f.rows = rows;
  f.warps = 1;
  while (f.warps * 2 * rows <= kWarps && (int64_t)f.warps * 64 * least < K) f.warps *= 2;
  const int64_t lanes = (int64_t)64 * f.warps * ((K + (int64_t)64 * f.warps * kLongest - 1) / ((int64_t)64 * f.warps * kLongest));      // segments there is room for
  f.seg = ((int)(((K + lanes - 1) / lanes + piece - 1) / piece) | 1) * piece;
  const int n_seg = (K + f.seg - 1) / f.seg;
  f.pitch = n_seg * f.seg * elem;
  f.pitch += (f.pitch & 16) ? 0 : 16;
  f.smem = (int64_t)rows * (f.pitch + (n_seg | 1) * 16 + (n_seg + 31) / 32 * 4) + f.seg * elem;
  f.grid = (n + rows - 1) / rows;
  return f;
}
// Where this kernel is the faster one: from more than 1024 columns on (512 3.9 4.8, 1024 5.5 5.2 to 9.0 9.8: us, staged or by the ring and so) as long as all CTAs are on the SMs in one
// round, and in more rounds the longer the chain is that the others have to wait for.  Its time over theirs, 1 / 300 / 888 / 1776 / 2400 / 3552 rows of bf16: 1056 columns 0.90 0.88 0.91 0.95
// 1.08 1.05, 1152 0.87 0.89 0.88 0.94 1.04 1.03, 1280 0.84 0.83 0.84 0.89 1.01 0.97, 1536 0.76 0.75 0.76 0.80 0.91 0.89, 2048 0.65 0.74 0.80 0.84 0.97 0.96, 4096 0.48 0.54 0.62 0.75 0.85 0.81;
// 8192 (two and three rounds) 0.33 0.38 0.48 0.61 0.92 0.97, 12288 0.25 0.31 0.40 0.69 0.87, 16384 0.21 0.28 0.37 0.64 0.85 1.00.  So eight rows to a CTA, above 1776 of them, from more than 1280 columns on.
// fp32, four rows to a CTA at most: 1056 columns 0.92 0.87 0.89 0.90, 4096 0.43 0.44 0.50 0.63, 16384 0.19 0.24 0.43 0.77; eight are level (2048 columns, 2200 rows 16.4 16.7; 3000 17.8 17.7).
static bool pays(int64_t n, int K, bool bf16, int64_t sms, Shape& f) {
  if (K <= 1024 || K > (1 << 17)) return false;
  f = shape(n, K, bf16, 1);
  while (f.grid > sms * kCtasPerSm && f.rows < (bf16 ? kMaxRows : kMaxRows / 2)) {
    const Shape two = shape(n, K, bf16, 2 * f.rows);
    if (two.smem + kStatic / 2 + kReserved > kSmem / kCtasPerSm) break;
    f = two;
  }
  if (f.rows == kMaxRows && K <= 1280) return false;
  const int64_t per_sm = std::min<int64_t>(kCtasPerSm, kSmem / (f.smem + kStatic / 2 + kReserved));
  return per_sm > 0 && f.grid <= per_sm * sms * std::max(1, K / 4096);
}
}  // namespace rms_seg
template <int FMT, bool BF16IN, bool UNIT, bool STOPS>
__global__ void __launch_bounds__(rms_seg::kThreads, rms_seg::kCtasPerSm)
rmsnorm_quantize_segments_kernel(const uint8_t* __restrict__ x, int64_t rows, int K, int rows_per_cta, int seg, int warps_per_row, int row_pitch,
                                 const float* __restrict__ gamma, float eps, uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, int* status, int stop) {
  using namespace rms_seg;
  extern __shared__ __align__(16) uint8_t seg_smem[];                   // rows | a segment of zeros | segments' gains | ends of runs
  __shared__ float rms_row[kMaxRows], warp_total[kWarps];
  __shared__ uint64_t full[kMaxRows];
  constexpr int kElem = BF16IN ? 2 : 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_seg = (K + seg - 1) / seg, seg_bytes = seg * kElem, gain_pitch = (n_seg | 1) * 16, masks = (n_seg + 31) / 32;
  const int row_bytes = K * kElem;
  uint8_t* const zeros = seg_smem + rows_per_cta * row_pitch;
  uint8_t* const gains = zeros + seg_bytes;
  uint32_t* const ends = reinterpret_cast<uint32_t*>(gains + rows_per_cta * gain_pitch);
  const int64_t row0 = (int64_t)blockIdx.x * rows_per_cta;
  const int n_rows = (int)min((int64_t)rows_per_cta, rows - row0);
  if (threadIdx.x < n_rows) mbar_init(&full[threadIdx.x], 1);
  fence_barrier_init();
  for (int r = warp; r < n_rows; r += kWarps)                           // zeros from the end of a row to the end of its last segment
    for (int i = row_bytes + lane * 16; i < n_seg * seg_bytes; i += 512) *reinterpret_cast<uint4*>(seg_smem + r * row_pitch + i) = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x * 16; i < seg_bytes; i += kThreads * 16) *reinterpret_cast<uint4*>(zeros + i) = make_uint4(0, 0, 0, 0);
  __syncthreads();
  grid_dependency_wait();
  grid_dependents_launch();
  const int asked = STOPS && stop == 2 ? n_rows / 2 : n_rows;           // test hook: the warp that asks for the rows stops half way
  if (warp == 0 && lane < asked) {
    mbar_arrive_expect_tx(&full[lane], (uint32_t)row_bytes);
    bulk_load_1d(seg_smem + lane * row_pitch, x + (row0 + lane) * row_bytes, (uint32_t)row_bytes, &full[lane]);
  }
  auto wait = [&](uint64_t* bar) -> bool {                              // bounded by 2^19 polls, about two seconds
#pragma unroll 1
    for (int it = 0; it < 1 << 19; ++it)
      if (mbar_try_wait<2000>(bar, 0)) return true;
    return false;
  };
  // step(v, i) for the elements (bf16) or squares (fp32) of two segments, in order
  auto walk = [&](const uint8_t* pa, const uint8_t* pb, auto&& step) {
#pragma unroll 1
    for (int j = 0; j < seg_bytes; j += 16) {
      const uint4 qa = *reinterpret_cast<const uint4*>(pa + j), qb = *reinterpret_cast<const uint4*>(pb + j);
      const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (BF16IN) {
          step(pair_u32(wa[i] << 16, wb[i] << 16), 0);
          step(pair_u32(wa[i] & 0xFFFF0000u, wb[i] & 0xFFFF0000u), 1);
        } else {
          const float fa = __uint_as_float(wa[i]), fb = __uint_as_float(wb[i]);
          step(pair_f32(__fmul_rn(fa, fa), __fmul_rn(fb, fb)), i & 1);
        }
      }
    }
  };
  auto add_square = [](uint64_t v, uint64_t c) { return BF16IN ? fma_sq_f32x2(v, c) : add_f32x2(c, v); };
  const int part = warp % warps_per_row, n_groups = kWarps / warps_per_row;
  const int per_part = ((n_seg + warps_per_row - 1) / warps_per_row + 63) / 64 * 64;   // segments of a warp, in groups of 64
  bool ok = true;
  for (int r0 = 0; r0 < n_rows; r0 += n_groups) {                       // (one pass where several warps share a row)
    const int r = r0 + warp / warps_per_row;
    const bool mine = r < n_rows;
    const uint8_t* row = seg_smem + r * row_pitch;
    if (mine && ok) ok = __all_sync(0xffffffffu, !(STOPS && stop == 1 && r >= n_rows / 2) && wait(&full[r]));
    const bool go = mine && ok;
    const int s_begin = part * per_part, s_end = min(n_seg, s_begin + per_part);
    auto segment = [&](int s) -> const uint8_t* { return s < s_end ? row + s * seg_bytes : zeros; };
    auto add_up = [&](int s0, float& sa, float& sb) {                   // about the sums of segments s0 + lane and s0 + 32 + lane
      uint64_t s[2] = {0, 0};
      walk(segment(s0 + lane), segment(s0 + 32 + lane), [&](uint64_t v, int which) { s[which] = add_square(v, s[which]); });
      unpair_f32(add_f32x2(s[0], s[1]), sa, sb);
    };
    float carry = 0.0f;                                                 // about the sum of what lies before
    if (warps_per_row > 1) {
      float total = 0.0f;
      if (go)
        for (int s0 = s_begin; s0 < s_end; s0 += 64) { float sa, sb; add_up(s0, sa, sb); total += sa + sb; }
#pragma unroll
      for (int o = 16; o > 0; o /= 2) total += __shfl_xor_sync(0xffffffffu, total, o);
      if (lane == 0) warp_total[warp] = total;
      __syncthreads();
      for (int w = warp - part; w < warp; ++w) carry += warp_total[w];
    }
    if (!go) continue;
    for (int s0 = s_begin; s0 < s_end; s0 += 64) {
      float sum[2], upto[2];
      add_up(s0, sum[0], sum[1]);
      upto[0] = sum[0];
      upto[1] = sum[1];
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const float ua = __shfl_up_sync(0xffffffffu, upto[0], o), ub = __shfl_up_sync(0xffffffffu, upto[1], o);
        if (lane >= o) { upto[0] += ua; upto[1] += ub; }
      }
      const float all_a = __shfl_sync(0xffffffffu, upto[0], 31), all_b = __shfl_sync(0xffffffffu, upto[1], 31);
      uint32_t e[2], even[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float end = (h ? carry + all_a : carry) + upto[h], begin = end - sum[h];
        constexpr float kMargin = 1.0f / 8192;                          // more than the sums in two orders differ by
        const uint32_t lo = __float_as_uint(begin * (1.0f - kMargin)) >> 23, hi = __float_as_uint(end * (1.0f + kMargin)) >> 23;
        e[h] = sum[h] == 0.0f && begin == 0.0f ? 0u : lo == hi && lo >= 40 && lo < 255 ? lo : kMarked;
        even[h] = (lo & 0xFFu) << 23;
      }
      carry += all_a + all_b;
      uint64_t ce = pair_u32(even[0], even[1]), co = pair_u32(even[0] | 1u, even[1] | 1u);
      walk(segment(s0 + lane), segment(s0 + 32 + lane), [&](uint64_t v, int) { ce = add_square(v, ce); co = add_square(v, co); });
      uint32_t end_even[2], end_odd[2];
      unpair_u32(ce, end_even[0], end_even[1]);
      unpair_u32(co, end_odd[0], end_odd[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // A gain that leaves the binade does so from any start; kept small, the gains of 32 segments fit.
        constexpr uint32_t kLeaves = 1u << 24;
        uint32_t d0 = min(end_even[h] - even[h], kLeaves), d1 = min(end_odd[h] - (even[h] | 1u), kLeaves);
        const uint32_t before = __shfl_up_sync(0xffffffffu, e[h], 1);
        const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || before != e[h]);
        const int head = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {                               // gains from the head of the run to this segment
          const uint32_t f0 = __shfl_up_sync(0xffffffffu, d0, o), f1 = __shfl_up_sync(0xffffffffu, d1, o);
          if (lane - o >= head) {
            const uint32_t g0 = d0, g1 = d1;
            d0 = f0 + ((f0 & 1u) ? g1 : g0);
            d1 = f1 + ((f1 & 1u) ? g0 : g1);
          }
        }
        const int s = s0 + 32 * h + lane, n_here = min(32, s_end - s0 - 32 * h);
        if (s < s_end) *reinterpret_cast<uint4*>(gains + r * gain_pitch + s * 16) = make_uint4(e[h], d0, d1, 0u);
        if (lane == 0 && n_here > 0) ends[r * masks + (s >> 5)] = (heads >> 1) | (1u << (n_here - 1));
      }
    }
  }
  if (__syncthreads_or(!ok)) {
    // the copies under way before shared memory goes to another CTA
    for (int r = 0; r < asked; ++r) wait(&full[r]);
    if (threadIdx.x == 0) atomicCAS(status, 0, 602);
    return;
  }
  if (warp == 0) {
    const int r = min(lane, n_rows - 1);
    const uint8_t* row = seg_smem + r * row_pitch;
    const uint4* gain = reinterpret_cast<const uint4*>(gains + r * gain_pitch);
    float ss = 0.0f;
    int i = 0, last = -1;                                               // segments that are in the sum; last segment of the next run
    uint32_t left = ends[r * masks];
    while (true) {
      bool stuck = false;
#pragma unroll 1
      while (i < n_seg && !stuck) {
        if (left == 0) left = ends[r * masks + (i >> 5)];
        last = (i & ~31) + __ffs(left) - 1;
        left &= left - 1;
        const uint4 q = gain[last];
        const uint32_t bits = __float_as_uint(ss), next = bits + ((bits & 1u) ? q.z : q.y);
        stuck = (bits >> 23) != q.x || (next >> 23) != q.x;
        if (!stuck) { ss = __uint_as_float(next); i = last + 1; }
      }
      if (__all_sync(0xffffffffu, i >= n_seg)) break;
      if (stuck) {                                                      // segments i to last as they lie
        const uint4* p = reinterpret_cast<const uint4*>(row + i * seg_bytes);
        const int n = (last + 1 - i) * (seg_bytes / 16);
        auto add = [&](const uint4& q) {
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (BF16IN) {
              const float lo = __uint_as_float(w[k] << 16), hi = __uint_as_float(w[k] & 0xFFFF0000u);
              ss = __fadd_rn(ss, __fmul_rn(lo, lo));
              ss = __fadd_rn(ss, __fmul_rn(hi, hi));
            } else {
              ss = __fadd_rn(ss, __fmul_rn(__uint_as_float(w[k]), __uint_as_float(w[k])));
            }
          }
        };
        uint4 ahead[4];                                                 // four pieces at a time, the next four under way
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < n) ahead[k] = p[k];
        int j = 0;
#pragma unroll 1
        for (; j + 4 <= n; j += 4) {
          const uint4 now[4] = {ahead[0], ahead[1], ahead[2], ahead[3]};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (j + 4 + k < n) ahead[k] = p[j + 4 + k];
#pragma unroll
          for (int k = 0; k < 4; ++k) add(now[k]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (j + k < n) add(ahead[k]);
        i = last + 1;
      }
      __syncwarp();
    }
    if (lane < n_rows) rms_row[lane] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)K), eps)));
  }
  __syncthreads();
  // y = (x rms) gamma, quantized: a warp keeps 512 columns (16 per lane, 2 lanes per block) and walks the rows; with fewer column units than warps several share one
  const int units = (K + 511) / 512, parts = max(1, kWarps / units), first = warp / units;
  uint8_t* const scale_bytes = gains;                                   // n_rows K / 32 bytes, less than the gains took
  auto quantize_rows = [&](auto cold_tag) -> bool {
    constexpr bool COLD = decltype(cold_tag)::value;
    bool finite = true;
    if (first >= parts) return finite;
    for (int u = warp - first * units; u < units; u += kWarps) {
      const int col = u * 512 + lane * 16;
      if (col >= K) continue;                                           // whole 2-lane groups: K % 32 == 0
      float g[2][8];
      widen8<false>(load_raw8<false, 16>(reinterpret_cast<const uint8_t*>(gamma + col)), g[0]);
      widen8<false>(load_raw8<false, 16>(reinterpret_cast<const uint8_t*>(gamma + col + 8)), g[1]);
      const uint8_t* src = seg_smem + first * row_pitch + col * kElem;
      uint8_t* dst = codes + (row0 + first) * K + col;
      uint8_t* sdst = scale_bytes + first * (K / 32) + col / 32;
#pragma unroll 1
      for (int r = first; r < n_rows; r += parts) {
        Raw8<BF16IN> raw[2];
        load_pair<BF16IN, kPieceShared>(raw, src, false);
        const float rms = rms_row[r];
        float v[2][8];
        widen8<BF16IN>(raw[0], v[0]);
        widen8<BF16IN>(raw[1], v[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 8; j += 2)
            unpair_f32(mul_f32x2(mul_f32x2(pair_f32(v[h][j], v[h][j + 1]), pair_f32(rms, rms)), pair_f32(g[h][j], g[h][j + 1])), v[h][j], v[h][j + 1]);
        uint32_t scode;
        uint2 w[2];
        finite &= quantize_lanes<FMT, UNIT, 2, COLD, true>(v, lane, w, scode);
        __stcs(reinterpret_cast<uint4*>(dst), make_uint4(w[0].x, w[0].y, w[1].x, w[1].y));
        if ((lane & 1) == 0) *sdst = (uint8_t)scode;
        src += parts * row_pitch;
        dst += (int64_t)parts * K;
        sdst += parts * (K / 32);
      }
    }
    return finite;
  };
  if (__syncthreads_or(!quantize_rows(std::false_type{}))) { quantize_rows(std::true_type{}); __syncthreads(); }
  const int n = n_rows * (K / 32);                                      // contiguous in memory, as the CTA's rows are
  uint8_t* out = scales + row0 * (K / 32);
  if ((reinterpret_cast<uintptr_t>(out) & 3) == 0 && (n & 3) == 0) {
    for (int i = threadIdx.x; i < n / 4; i += kThreads) reinterpret_cast<uint32_t*>(out)[i] = reinterpret_cast<const uint32_t*>(scale_bytes)[i];
  } else {
    for (int i = threadIdx.x; i < n; i += kThreads) out[i] = scale_bytes[i];
  }
}

// Append one token to a KV cache: row pos[b] of every (batch, KV head) of K and of V is quantized (blocks of 32
// along d, same rule and same code path as quantize_rows_kernel) and written in place.  chunk = 8 consecutive
// elements of one new row; 4 consecutive lanes = one block.  A position outside [0, L) is skipped.
// A step of one sequence is a chain of latencies: the row, column and sequence of a thread are worked out while the kernel before still runs (K in one half of
// the grid, V in the other, 32-bit divisions), and the position is asked for with the values, not after them: one sequence of 6000 keys 12.4 -> 11.8 us a step.
template <int FMT>
__global__ void __launch_bounds__(128) kv_append_kernel(const float* __restrict__ k_new, const float* __restrict__ v_new,
                                                        uint32_t rows, uint32_t H_kv, int L, uint32_t d, const int32_t* __restrict__ pos,
                                                        uint8_t* __restrict__ k_codes, uint8_t* __restrict__ k_scales,
                                                        uint8_t* __restrict__ v_codes, uint8_t* __restrict__ v_scales) {
  const uint32_t cpr = d / 8, nchunks = rows * cpr;          // chunks per row (a multiple of 4), of K and of V
  const float* const src = blockIdx.y ? v_new : k_new;
  uint8_t* const codes = blockIdx.y ? v_codes : k_codes;
  uint8_t* const scales = blockIdx.y ? v_scales : k_scales;
  const uint32_t lane = threadIdx.x & 31, stride = gridDim.x * blockDim.x;
  uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t row = c / cpr, col = (c - row * cpr) * 8, b = row / H_kv;       // of the first chunk, while the kernel before still runs
  grid_dependency_wait();
  grid_dependents_launch();
  for (; c - lane < nchunks; c += stride, row = c / cpr, col = (c - row * cpr) * 8, b = row / H_kv) {
    const bool live = c < nchunks;
    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
    int at = -1;
    if (live) {                                              // both latencies at once
      const float4* q = reinterpret_cast<const float4*>(src + (size_t)row * d + col);
      v0 = q[0]; v1 = q[1];
      at = pos[b];
    }
    const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    float amax = 0.0f, nonfinite = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) { amax = fmaxf(amax, fabsf(v[j])); nonfinite = fmaf(v[j], 0.0f, nonfinite); }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    if (at < 0 || at >= L) continue;
    uint32_t scode = 0; float p2 = 1.0f;
    if (amax > 0.0f) block_scale<FMT>(amax, scode, p2);
    uint32_t w0, w1;
    if (nonfinite == 0.0f) {
      w0 = hw_encode4<FMT>(v[0] * p2, v[1] * p2, v[2] * p2, v[3] * p2);
      w1 = hw_encode4<FMT>(v[4] * p2, v[5] * p2, v[6] * p2, v[7] * p2);
    } else {
      w0 = ref_encode4<FMT>(v[0] * p2, v[1] * p2, v[2] * p2, v[3] * p2);
      w1 = ref_encode4<FMT>(v[4] * p2, v[5] * p2, v[6] * p2, v[7] * p2);
    }
    const int64_t crow = (int64_t)row * L + at;               // row of the cache
    *reinterpret_cast<uint2*>(codes + crow * d + col) = make_uint2(w0, w1);
    if ((col & 31) == 0) scales[crow * (d / 32) + col / 32] = (uint8_t)scode;
  }
}

// One warp = 32 rows x 32 columns, a lane = 8 of the rows x 4 adjacent columns in registers, all its loads in flight, 128 bytes
// of a row per request; the four lanes of a column group end up with the maximum of one column each and hand its factor back.
// HBM bound; x is read once.  67 M elements: 102 us with a thread per column group (32 rows one after the other, read twice),
// 65 us now.
// ATOMS: scales go to the scale-factor atoms [batch][ceil(rows/128)][ceil(cols/128)][512] (byte = column n of the
// chunk, 32-key block kbi of the tile) instead of row-major [batch][ceil(rows/32)][cols].
template <int FMT, bool ATOMS = false>
__global__ void __launch_bounds__(128) quantize_keys_kernel(const float* __restrict__ x, int64_t batch, int64_t rows,
                                                            int64_t cols, uint8_t* __restrict__ codes,
                                                            uint8_t* __restrict__ scales) {
  const int lane = threadIdx.x & 31, r0 = (lane >> 3) * 8;
  const bool h16 = lane & 16, h8 = lane & 8;
  const int64_t ncb = (cols + 31) / 32, nkb = (rows + 31) / 32, units = batch * nkb * ncb;
  grid_dependency_wait();
  grid_dependents_launch();
  for (int64_t u = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); u < units; u += (int64_t)gridDim.x * 4) {
    int64_t cb, kb, bt;
    if (units < (int64_t)1 << 31) {                                // 32-bit divisions whenever the index fits
      const uint32_t q = (uint32_t)u / (uint32_t)ncb, b32 = q / (uint32_t)nkb;
      cb = (uint32_t)u - q * (uint32_t)ncb;
      kb = q - b32 * (uint32_t)nkb;
      bt = b32;
    } else {
      cb = u % ncb; kb = u / ncb % nkb; bt = u / (ncb * nkb);
    }
    const int64_t col = cb * 32 + (lane & 7) * 4, row = bt * rows + kb * 32 + r0;
    const int n = col < cols ? (int)min((int64_t)8, rows - kb * 32 - r0) : 0;   // rows of this lane
    const float* src = x + row * cols + col;
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < n ? __ldcs(reinterpret_cast<const float4*>(src + i * cols)) : make_float4(0.f, 0.f, 0.f, 0.f);
    float m[4] = {0.f, 0.f, 0.f, 0.f};
    float nonfinite = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      m[0] = fmaxf(m[0], fabsf(v[i].x)); m[1] = fmaxf(m[1], fabsf(v[i].y));
      m[2] = fmaxf(m[2], fabsf(v[i].z)); m[3] = fmaxf(m[3], fabsf(v[i].w));
      nonfinite = fmaf(v[i].x, 0.0f, fmaf(v[i].y, 0.0f, fmaf(v[i].z, 0.0f, fmaf(v[i].w, 0.0f, nonfinite))));
    }
    const float a = fmaxf(h16 ? m[2] : m[0], __shfl_xor_sync(0xffffffffu, h16 ? m[0] : m[2], 16));
    const float c = fmaxf(h16 ? m[3] : m[1], __shfl_xor_sync(0xffffffffu, h16 ? m[1] : m[3], 16));
    const float amax = fmaxf(h8 ? c : a, __shfl_xor_sync(0xffffffffu, h8 ? a : c, 8));   // of column lane / 8 of the four
    uint32_t sc = 0;
    float p2 = 1.0f, f[4];
    if (amax > 0.0f) block_scale<FMT>(amax, sc, p2);
#pragma unroll
    for (int q = 0; q < 4; ++q) f[q] = __shfl_sync(0xffffffffu, p2, (lane & 7) + 8 * q);
    uint8_t* dst = codes + row * cols + col;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t w = (nonfinite == 0.0f) ? hw_encode4<FMT>(v[i].x * f[0], v[i].y * f[1], v[i].z * f[2], v[i].w * f[3])
                                             : ref_encode4<FMT>(v[i].x * f[0], v[i].y * f[1], v[i].z * f[2], v[i].w * f[3]);
      if (i < n) __stcs(reinterpret_cast<uint32_t*>(dst + i * cols), w);
    }
    const int64_t mine = col + (lane >> 3);
    if (col < cols) {
      if (!ATOMS) scales[(bt * nkb + kb) * cols + mine] = (uint8_t)sc;
      else scales[((bt * ((rows + 127) / 128) + kb / 4) * ((cols + 127) / 128) + mine / 128) * 512 + sf_atom_offset((int)(mine & 127), (int)(kb & 3))] = (uint8_t)sc;
    }
  }
}

// Scale-factor atoms [batch][ntile][dch][512] from the other layouts of block scales: one warp per atom, a lane writes the 16 bytes of rows or columns lane,
// lane + 32, + 64 and + 96; rows, columns and blocks past the edge get code 0x7F = 2^0.  (A thread per row or column, with the divisions that find its place, was a fifth
// of the time of the re-blocking kernel beside which the scales of Q and K are re-tiled: 8 x 16 heads of 4096, d = 128, 33.8 -> 31.6 us, 4 x 32 / 8 of 8192 22.2 -> 18.8, 2 x 16 / 8 of 8192, d = 256, 20.2 -> 18.5.
// Row-major and group-major scales in one loop, a row after the other: 8 / 2 heads of 640 keys, d = 128, group-major 12.6 -> 13.9 us a call, apart 11.9; 2 x 16 / 8 of 700, d = 256, 20.4, 21.2, 20.4.)
//   kRows   along d, row-major [batch][S][d/32]
//   kGroups along d, group-major [batch][d/32][S] (the reference's QK_A_scales_row[FA_GK][FA_SQ] per head,
//           kernels/flash_attention_mx/gen_data.py:82-83)
//   kKeys   along keys, row-major [batch][ceil(S/32)][d]
enum RetileKind { kRows = 0, kGroups = 1, kKeys = 2 };
RK_DEVINL void retile_atom(const RetileJob& job, int64_t atom, int64_t total) {
  const int64_t S = job.S, d = job.d;
  const int64_t nbd = d / 32, nkb = (S + 31) / 32, ntile = (S + 127) / 128, dch = (d + 127) / 128;
  const int lane = threadIdx.x & 31;
  uint8_t* const out = job.out + atom * 512;
  int64_t ch, tile, bt;
  if (total < (int64_t)1 << 31) {           // 32-bit divisions whenever the index fits
    const uint32_t a32 = (uint32_t)atom, q = dch == 1 ? a32 : a32 / (uint32_t)dch;
    ch = a32 - q * (uint32_t)dch;
    const uint32_t b32 = q / (uint32_t)ntile;
    tile = q - b32 * (uint32_t)ntile;
    bt = b32;
  } else {
    ch = atom % dch; tile = (atom / dch) % ntile; bt = atom / (dch * ntile);
  }
  uint32_t w[4];
  if (job.kind == kKeys) {                  // four adjacent columns of the four key blocks, turned
    const int64_t col = ch * 128 + lane * 4;
    key_scale_words(job.in + (bt * nkb + tile * 4) * d + col, d, (int)min((int64_t)4, nkb - tile * 4), col < d, (reinterpret_cast<uintptr_t>(job.in) & 3) == 0, w);      // (d is a multiple of 32)
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint32_t*>(out + sf_atom_offset(lane * 4 + i, 0)) = w[i];
    return;
  }
  const int64_t row = tile * 128 + lane;
  if (job.kind == kRows) {
    row_scale_words(job.in + (bt * S + row) * nbd + ch * 4, job.in, nbd, (int)min((int64_t)128, S - row), (int)min((int64_t)4, nbd - ch * 4), w);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = 0x7F7F7F7Fu;
      if (row + i * 32 < S) {
        w[i] = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int64_t blk = ch * 4 + k;
          w[i] |= (blk < nbd ? (uint32_t)job.in[(bt * nbd + blk) * S + row + i * 32] : 0x7Fu) << (8 * k);
        }
      }
    }
  }
  *reinterpret_cast<uint4*>(out + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
}
__host__ __device__ inline int64_t retile_atoms(const RetileJob& job) { return job.batch * ((job.S + 127) / 128) * ((job.d + 127) / 128); }
// The jobs of a prefill call ride along with whichever preparation kernel it needs anyway (a launch costs more than they do):
// its first jobs.ctas CTAs do them, true for those.  The atoms of all jobs in a row, so that a small call has one for each warp at most.
RK_DEVINL bool retile_jobs(const RetileJobs& jobs) {
  if ((int)blockIdx.x >= jobs.ctas) return false;
  const int64_t warps = (int64_t)jobs.ctas * (blockDim.x / 32);
  int64_t at = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
#pragma unroll 1
  for (int i = 0; i < jobs.n; ++i) {
    const int64_t n = retile_atoms(jobs.job[i]);
#pragma unroll 1
    for (; at < n; at += warps) retile_atom(jobs.job[i], at, n);
    at -= n;
  }
  return true;
}
__global__ void __launch_bounds__(128) retile_scales_kernel(const RetileJobs jobs) {
  grid_dependency_wait();
  grid_dependents_launch();
  retile_jobs(jobs);
}

// ---- V re-blocking: scales along d -> MX blocks along the keys (rk_rebase.cuh) ---------------------------------------
// A CTA = 128 keys x 8 NC columns at a time, a warp = 32 of the keys, a lane = 8 of them x NC adjacent columns, all its loads
// in flight; the column maxima meet by the shuffles of a reduce-scatter.  NC = 8, or 4 where the codes are not 8-byte aligned.
// 67 M codes E4M3: 53 us in integer arithmetic on the codes (12 instructions per code, 16 warps per SM, rows with a zero or
// subnormal code on a path of their own), 31.6 us here beside the scales' re-tiling.  (All columns of 128 keys by one CTA: 30.4, but 33.5 M codes 18.8 -> 19.8 and calls of few
// keys 0.2 us more.  On the codes as bytes, where a power of two is a step of 8: 35 us, and 55 with the words done again in which a code is or becomes subnormal.)
// Idx: of an element within 32 rows; int64_t where these are longer than 2^31 bytes (for all calls: 33.5 M codes 13.6 -> 13.9 us).
constexpr int kRebaseThreads = 128;
template <int FMT, bool TILED, int NC, class Idx = int>
__global__ void __launch_bounds__(kRebaseThreads, 7) rebase_v_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ scales,
                                                                 int64_t batch, int64_t S, int64_t d, uint8_t* __restrict__ out_codes,
                                                                 uint8_t* __restrict__ out_scales, const RetileJobs jobs) {
  constexpr int NW = NC / 4, NB = NC / 4, CP = NC / 4;             // words per key of a thread; 32-column blocks of a warp; columns whose scales a thread works out
  __shared__ __align__(4) uint8_t sc_sm[8 * NC * 4];
  __shared__ __align__(16) uint32_t fac_sm[kRebaseThreads / 32][NB][32];
  grid_dependency_wait();
  grid_dependents_launch();
  if (retile_jobs(jobs)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nkb = (S + 31) / 32, nbd = d / 32, ntile = (S + 127) / 128, dch = (d + 127) / 128;
  const int64_t cun = TILED ? dch * (16 / NC) : (d + 8 * NC - 1) / (8 * NC), units = batch * ntile * cun, stride = gridDim.x - jobs.ctas;
  for (int64_t u = (int64_t)blockIdx.x - jobs.ctas; u < units; u += stride) {
    int64_t cu, kt, bt;
    if (units < (int64_t)1 << 31) {                                // 32-bit divisions whenever the index fits
      const uint32_t q = (uint32_t)u / (uint32_t)cun;
      cu = (uint32_t)u - q * (uint32_t)cun;
      const uint32_t b32 = q / (uint32_t)ntile;
      kt = q - b32 * (uint32_t)ntile;
      bt = b32;
    } else {
      cu = u % cun; kt = u / cun % ntile; bt = u / (cun * ntile);
    }
    const int64_t kb = kt * 4 + warp;
    const int64_t row0 = bt * S + kb * 32, col = cu * 8 * NC + (lane & 7) * NC;
    const int n = (int)max((int64_t)0, min((int64_t)32, S - kb * 32));   // keys of this block that exist
    const bool in = col < d && n > 0;
    uint32_t sc[CP];
    uint8_t* const dst = out_codes + row0 * d + col;
    const Idx di = (Idx)d;
    rebase_block<FMT, NC, false, Idx>(codes + row0 * d, scales + row0 * nbd, di, (Idx)cu, n, fac_sm[warp], lane,
                                      [=](int k, const uint32_t (&o)[NW]) {
                                        if (NC == 8) *reinterpret_cast<uint2*>(dst + k * di) = make_uint2(o[0], o[NW - 1]);
                                        else *reinterpret_cast<uint32_t*>(dst + k * di) = o[0];
                                      },
                                      [=](int k, int c, uint8_t code) { dst[k * di + c] = code; }, sc);
    if (TILED) {
      // the four warps' scale bytes of a column are one word of its atom
#pragma unroll
      for (int h = 0; h < CP; ++h) sc_sm[((lane & 7) * NC + (lane >> 3) * CP + h) * 4 + warp] = (uint8_t)sc[h];
      __syncthreads();
      for (int c = threadIdx.x; c < 8 * NC; c += kRebaseThreads) {
        const int64_t n128 = cu * 8 * NC + c;
        *reinterpret_cast<uint32_t*>(out_scales + ((bt * ntile + kt) * dch + n128 / 128) * 512 + sf_atom_offset((int)(n128 % 128), 0)) =
            *reinterpret_cast<const uint32_t*>(sc_sm + c * 4);
      }
      __syncthreads();
    } else if (in) {
#pragma unroll
      for (int h = 0; h < CP; ++h) out_scales[(bt * nkb + kb) * d + col + (lane >> 3) * CP + h] = (uint8_t)sc[h];
    }
  }
}

// The reference's streaming K operand (kernels/flash_attention_mx_gqa/fa_gen_data.py:110-117): per KV head and key
// block j a transposed tile K^T [d][Bk] (QK_B_blocks) with group-major scales [d/32][Bk] (QK_B_scales_blocks)
// -> natural K codes [heads][nblk*Bk][d] and row-major scales [heads][nblk*Bk][d/32].
// One CTA transposes a 32 x 32 byte tile through shared memory; scales by one thread per output byte.
__global__ void __launch_bounds__(256) import_kt_blocks_kernel(const uint8_t* __restrict__ kt, const uint8_t* __restrict__ kts,
                                                               int64_t heads, int nblk, int Bk, int d,
                                                               uint8_t* __restrict__ k, uint8_t* __restrict__ ks) {
  __shared__ uint8_t tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;           // 32 x 8
  const int64_t tiles_k = Bk / 32, tiles_d = d / 32;
  const int64_t ntiles = heads * nblk * tiles_d * tiles_k;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t tk = t % tiles_k, td = (t / tiles_k) % tiles_d, blk = t / (tiles_k * tiles_d);   // blk = head * nblk + j
    const uint8_t* src = kt + (blk * d + td * 32) * Bk + tk * 32;    // rows = d index, cols = key inside the block
#pragma unroll
    for (int i = 0; i < 4; ++i) tile[ty + 8 * i][tx] = src[(int64_t)(ty + 8 * i) * Bk + tx];
    __syncthreads();
    uint8_t* dst = k + (blk * Bk + tk * 32) * d + td * 32;            // rows = key, cols = d index
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[(int64_t)(ty + 8 * i) * d + tx] = tile[tx][ty + 8 * i];
    __syncthreads();
  }
  const int nbd = d / 32;
  const int64_t nsc = heads * nblk * (int64_t)Bk * nbd;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nsc; t += (int64_t)gridDim.x * blockDim.x) {
    const int g = (int)(t % nbd);
    const int64_t key = (t / nbd) % Bk, blk = t / ((int64_t)nbd * Bk);
    ks[t] = kts[(blk * nbd + g) * Bk + key];
  }
}

// ---- dense 6- and 4-bit operands -------------------------------------------------------------------------------------
// four byte codes -> BITS * 4 bits, code i at bits [BITS * i, BITS * i + BITS)
template <int BITS> RK_DEVINL uint32_t pack4(uint32_t w) {
  if (BITS == 4) {
    w = (w & 0x000F000Fu) | ((w >> 4) & 0x00F000F0u);
    return (w & 0xFFu) | ((w >> 8) & 0xFF00u);
  }
  w = (w & 0x003F003Fu) | ((w >> 2) & 0x0FC00FC0u);
  return (w & 0xFFFu) | ((w >> 4) & 0xFFF000u);
}
// groups of four packed codes -> 32-bit words in order (the order TMA's 16U6_ALIGN16B / 16U4_ALIGN16B types expand from):
// N groups of 24 bits -> 3 N / 4 words, or of 16 bits -> N / 2 words
template <int BITS, int N> RK_DEVINL void join_groups(const uint32_t (&c)[N], uint32_t (&w)[N * BITS / 8]) {
  if (BITS == 4) {
#pragma unroll
    for (int i = 0; i < N / 2; ++i) w[i] = c[2 * i] | (c[2 * i + 1] << 16);
  } else {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      w[3 * i] = c[4 * i] | (c[4 * i + 1] << 24);
      w[3 * i + 1] = (c[4 * i + 1] >> 8) | (c[4 * i + 2] << 16);
      w[3 * i + 2] = (c[4 * i + 2] >> 16) | (c[4 * i + 3] << 8);
    }
  }
}

// byte codes [rows][d] -> packed [rows][dp * BITS/8 bytes], dp = d rounded up to 128, padding codes 0.  A warp packs 512 codes at
// a time, 16 per lane, four times' loads in flight; the 6-bit words (12 bytes per lane) pass through shared memory to leave in
// 16-byte stores (one 16-byte load in flight and three 4-byte stores at a stride of 12 left HBM at a third of its rate).
template <int BITS> RK_DEVINL void pack_rows_body(const PackJob& job, int64_t d, int64_t dp, uint32_t* stage, int64_t warp0, int64_t warps) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const int64_t groups = dp / 16, total = job.rows * groups;          // a multiple of 8
  for (int64_t c0 = warp0 * 32; c0 < total; c0 += U * 32 * warps) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t t = c0 + u * 32 * warps + lane;
      v[u] = make_uint4(0u, 0u, 0u, 0u);
      if (t < total) {
        if (dp == d) {
          v[u] = __ldcs(reinterpret_cast<const uint4*>(job.in) + t);
        } else {
          const int64_t r = t / groups, g = t - r * groups;
          if (g * 16 < d) v[u] = __ldcs(reinterpret_cast<const uint4*>(job.in + r * d + g * 16));
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t first = c0 + u * 32 * warps;
      if (first >= total) break;
      const int n = (int)min((int64_t)32, total - first);             // lanes with codes
      const uint32_t c[4] = {pack4<BITS>(v[u].x), pack4<BITS>(v[u].y), pack4<BITS>(v[u].z), pack4<BITS>(v[u].w)};
      uint32_t w[BITS / 2];
      join_groups<BITS, 4>(c, w);
      if (BITS == 4) {
        if (lane < n) __stcs(reinterpret_cast<uint2*>(job.out) + first + lane, make_uint2(w[0], w[1]));
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) stage[lane * 3 + i] = w[i % (BITS / 2)];
        __syncwarp();
        if (lane < n * 3 / 4) __stcs(reinterpret_cast<uint4*>(job.out + first * 12) + lane, reinterpret_cast<const uint4*>(stage)[lane]);
        __syncwarp();
      }
    }
  }
}
__global__ void __launch_bounds__(256) pack_rows_kernel(const PackJobs packs, int64_t d, int64_t dp, const RetileJobs jobs) {
  __shared__ __align__(16) uint32_t stage[8][96];
  grid_dependency_wait();
  grid_dependents_launch();
  if (retile_jobs(jobs)) return;
  const int64_t warp0 = ((int64_t)blockIdx.x - jobs.ctas) * 8 + (threadIdx.x >> 5), warps = ((int64_t)gridDim.x - jobs.ctas) * 8;
#pragma unroll 1
  for (int i = 0; i < packs.n; ++i) {
    if (packs.job[i].bits == 4) pack_rows_body<4>(packs.job[i], d, dp, stage[threadIdx.x >> 5], warp0, warps);
    else pack_rows_body<6>(packs.job[i], d, dp, stage[threadIdx.x >> 5], warp0, warps);
  }
}

// V for the tensor core in a 6- or 4-bit format: byte codes [batch][S][d] -> packed transposed [batch][d][Sp * BITS/8], Sp = S
// rounded up to 128 (sub-byte operands may not be MN-major).  REBASE: V comes scaled along d and is re-blocked along the keys
// on the way (decode exactly, block rule down each column, encode: the same result as rebase_v_kernel), the new block scales
// going to the scale-factor atoms.
// One CTA = 128 keys x 128 columns, a warp = one 32-key block, a thread = 4 columns x 32 keys in registers, all its loads in
// flight.  As in the re-blocking kernel the codes go through f16; pairs of keys of one column go back through
// the converter in the order in which they are packed.  The packed words meet in shared memory and leave in 16-byte stores.
// 33.5 M codes E3M2: re-blocking 138 us and transposition 27 us as kernels of their own, 31 us here.  (Seven CTAs per SM: eight spill
// more registers, five and six leave too few loads in flight: 1 and 2 us slower.)
// codes of four consecutive keys, packed
template <int FMT> RK_DEVINL uint32_t encode_pack4(float a, float b, float c, float d) {
  uint32_t r;
  if (FMT == 4) {
    asm("{\n\t.reg .b8 l, h;\n\tcvt.rn.satfinite.e2m1x2.f32 l, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 h, %4, %3;\n\tmov.b32 %0, {l, h, l, h};\n\t}"
        : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
    return r & 0xFFFFu;
  }
  return pack4<6>(hw_encode4<FMT>(a, b, c, d));
}
template <int FMT, bool REBASE>
__global__ void __launch_bounds__(128, 7) pack_v_kernel(const uint8_t* __restrict__ in, const uint8_t* __restrict__ scales, int64_t S, int64_t d,
                                                     int64_t Sp, uint8_t* __restrict__ out, uint8_t* __restrict__ atoms) {
  constexpr int BITS = FMT == 4 ? 4 : 6, kWords = BITS, kRow = 4 * kWords, kPitch = kRow + 1;   // words per key block, per column; pitch
  __shared__ uint32_t buf[128 * kPitch];
  __shared__ __align__(16) uint32_t fac[4][128];             // [32-column block][key]: packed f16 2^(s - smax)
  __shared__ int smax_sm[4][4];                                  // [32-column block][key block], -1: the slow form
  const int lane = threadIdx.x & 31, kb = threadIdx.x >> 5;
  const int64_t ktiles = Sp / 128, dch = (d + 127) / 128, nbd = d / 32;
  const int64_t ch = blockIdx.x % dch, kt = blockIdx.x / dch % ktiles, bt = blockIdx.x / (dch * ktiles);
  const int64_t key0 = kt * 128 + kb * 32, col0 = ch * 128 + lane * 4;
  grid_dependency_wait();
  grid_dependents_launch();
  const int n = (int)max((int64_t)0, min((int64_t)32, S - key0));    // keys of this block that exist
  const uint8_t* src = in + (bt * S + key0) * d + col0;
  uint32_t w[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) w[k] = (k < n && col0 < d) ? __ldg(reinterpret_cast<const uint32_t*>(src + k * d)) : 0u;
  uint32_t packed[4][8];                                         // [column][groups of four keys]
  uint32_t code[4] = {0x7Fu, 0x7Fu, 0x7Fu, 0x7Fu};               // new scale codes; of columns and blocks that do not exist, 2^0
  if (REBASE) {
    const uint8_t* sk = scales + (bt * S + key0 + lane) * nbd + ch * 4;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const bool live = lane < n && ch * 4 + b < nbd;
      const int s = live ? (int)__ldg(sk + b) : -1;
      const int top = __reduce_max_sync(0xffffffffu, s), low = __reduce_min_sync(0xffffffffu, live ? s : 255);
      fac[b][kb * 32 + lane] = live ? (uint32_t)max(15 + s - top, 1) * 0x04000400u : 0u;
      if (lane == 0) smax_sm[b][kb] = (top < 0 || (low >= 20 && top <= 235 && top - low <= RebaseT<FMT>::kSpan)) ? max(top, 0) : -1;
    }
    __syncwarp();
    const int blk = lane >> 3, smax = smax_sm[blk][kb];
    if (smax >= 0) {
      uint32_t x[32], y[32], mx = 0u, my = 0u;                    // columns 0, 1 and 2, 3 of the thread
#pragma unroll
      for (int k = 0; k < 32; k += 4) {
        const uint4 f4 = *reinterpret_cast<const uint4*>(&fac[blk][kb * 32 + k]);
        const uint32_t f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t c = clean_codes<FMT>(w[k + e]);
          x[k + e] = hmul2(decode_f16x2<FMT>(c), f[e]);
          y[k + e] = hmul2(decode_f16x2<FMT>(c >> 16), f[e]);
          mx = max_u16x2(mx, x[k + e] & 0x7FFF7FFFu);
          my = max_u16x2(my, y[k + e] & 0x7FFF7FFFu);
        }
      }
      const float unit = __uint_as_float((uint32_t)smax << 23);                                     // 2^(smax - 127)
      const float am[4] = {f16_lo(mx) * unit, f16_hi(mx) * unit, f16_lo(my) * unit, f16_hi(my) * unit};
      float f[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t sc = 0; float p2 = 1.0f;
        if (am[q] > 0.0f) block_scale<FMT>(am[q], sc, p2);
        if (n > 0 && col0 < d) code[q] = sc;
        f[q] = unit * p2;
      }
#pragma unroll
      for (int k = 0; k < 32; k += 4) {
        packed[0][k / 4] = encode_pack4<FMT>(f16_lo(x[k]) * f[0], f16_lo(x[k + 1]) * f[0], f16_lo(x[k + 2]) * f[0], f16_lo(x[k + 3]) * f[0]);
        packed[1][k / 4] = encode_pack4<FMT>(f16_hi(x[k]) * f[1], f16_hi(x[k + 1]) * f[1], f16_hi(x[k + 2]) * f[1], f16_hi(x[k + 3]) * f[1]);
        packed[2][k / 4] = encode_pack4<FMT>(f16_lo(y[k]) * f[2], f16_lo(y[k + 1]) * f[2], f16_lo(y[k + 2]) * f[2], f16_lo(y[k + 3]) * f[2]);
        packed[3][k / 4] = encode_pack4<FMT>(f16_hi(y[k]) * f[3], f16_hi(y[k + 1]) * f[3], f16_hi(y[k + 2]) * f[3], f16_hi(y[k + 3]) * f[3]);
      }
    } else {
      // block scales far apart or near the ends of the range: through fp32, element by element
      const uint8_t* sb = scales + (bt * S + key0) * nbd + col0 / 32;
      float am[4] = {0.f, 0.f, 0.f, 0.f}, p2[4];
      for (int k = 0; k < n; ++k) {
        const uint32_t c = *reinterpret_cast<const uint32_t*>(src + k * d), s = sb[k * nbd];
#pragma unroll
        for (int q = 0; q < 4; ++q) am[q] = fmaxf(am[q], fabsf(decode_scaled<FMT>((c >> (8 * q)) & 0xFFu, s)));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) { code[q] = 0; p2[q] = 1.0f; if (am[q] > 0.0f) block_scale<FMT>(am[q], code[q], p2[q]); }
#pragma unroll
      for (int g = 0; g < 8; ++g)
#pragma unroll
        for (int q = 0; q < 4; ++q) packed[q][g] = 0u;
#pragma unroll 1
      for (int k = 0; k < n; ++k) {
        const uint32_t c = *reinterpret_cast<const uint32_t*>(src + k * d), s = sb[k * nbd];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t e = encode_rne<FMT>(decode_scaled<FMT>((c >> (8 * q)) & 0xFFu, s) * p2[q]) << (BITS * (k & 3));
#pragma unroll
          for (int g = 0; g < 8; ++g) packed[q][g] |= (k >> 2) == g ? e : 0u;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = lane * 4 + q;
      atoms[((bt * ktiles + kt) * dch + ch) * 512 + sf_atom_offset(c, kb)] = (uint8_t)code[q];
    }
  } else {
#pragma unroll
    for (int k = 0; k < 32; k += 4) {                               // 4 keys x 4 columns of bytes, transposed
      const uint32_t a = __byte_perm(w[k], w[k + 1], 0x5140), b = __byte_perm(w[k + 2], w[k + 3], 0x5140);
      const uint32_t c = __byte_perm(w[k], w[k + 1], 0x7362), e = __byte_perm(w[k + 2], w[k + 3], 0x7362);
      packed[0][k / 4] = pack4<BITS>(__byte_perm(a, b, 0x5410));
      packed[1][k / 4] = pack4<BITS>(__byte_perm(a, b, 0x7632));
      packed[2][k / 4] = pack4<BITS>(__byte_perm(c, e, 0x5410));
      packed[3][k / 4] = pack4<BITS>(__byte_perm(c, e, 0x7632));
    }
  }
  // word i of column c sits at (i + c / 32) % kRow: with the odd pitch a store of 32 lanes then touches all banks
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t o[kWords];
    join_groups<BITS, 8>(packed[q], o);
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      int at = kb * kWords + i + (lane >> 3);
      at -= at >= kRow ? kRow : 0;
      buf[(lane * 4 + q) * kPitch + at] = o[i];
    }
  }
  __syncthreads();
  const int cols = (int)min((int64_t)128, d - ch * 128);
  for (int i = threadIdx.x; i < cols * (kRow / 4); i += 128) {
    const int c = i / (kRow / 4), chunk = i - c * (kRow / 4);
    uint32_t v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      int at = chunk * 4 + e + (c >> 5);
      at -= at >= kRow ? kRow : 0;
      v[e] = buf[c * kPitch + at];
    }
    *reinterpret_cast<uint4*>(out + (bt * d + ch * 128 + c) * (Sp * BITS / 8) + kt * (kRow * 4) + chunk * 16) = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

static int grid_for(int64_t work_items, int threads, int per_sm) {
  const int64_t want = (work_items + threads - 1) / threads;
  const int64_t cap = (int64_t)num_sms() * per_sm;
  return (int)max((int64_t)1, min(want, cap));
}

#define RK_DISPATCH_FMT(fmt, ...)                  \
  switch (fmt) {                                   \
    case 0: { constexpr int F = 0; __VA_ARGS__; } break; \
    case 1: { constexpr int F = 1; __VA_ARGS__; } break; \
    case 2: { constexpr int F = 2; __VA_ARGS__; } break; \
    case 3: { constexpr int F = 3; __VA_ARGS__; } break; \
    case 4: { constexpr int F = 4; __VA_ARGS__; } break; \
    default: return RK_ERR_BAD_FORMAT;             \
  }

int launch_quantize_rows_bf16(const void* x, int64_t rows, int64_t cols, int fmt, uint8_t* codes, uint8_t* scales,
                              cudaStream_t st) {
  const int64_t nchunks = rows * cols / 8;
  if (nchunks == 0) return RK_OK;
  const int grid = grid_for(nchunks, 256, 8);
  RK_DISPATCH_FMT(fmt, return (int)launch_pdl(quantize_rows_kernel<F, true, 0>, dim3(grid), dim3(256), 0, st, reinterpret_cast<const float4*>(x),
                                              nchunks, reinterpret_cast<uint2*>(codes), scales, (int64_t)0, 0));
  return RK_OK;
}

// Blocks along d with a chosen scale layout (see quantize_rows_kernel); x is fp32 or bf16 [batch][S][d].
int launch_quantize_rows_ex(const void* x, bool bf16, int64_t batch, int64_t S, int64_t d, int fmt, uint8_t* codes,
                            uint8_t* scales, int layout, cudaStream_t st) {
  const int64_t nchunks = batch * S * d / 8;
  if (nchunks == 0) return RK_OK;
  const int grid = grid_for(nchunks, 256, 8);
  const float4* xp = reinterpret_cast<const float4*>(x);
  uint2* cp = reinterpret_cast<uint2*>(codes);
  const int nbd = (int)(d / 32);
#define RK_QX(BF, LAY) RK_DISPATCH_FMT(fmt, return (int)launch_pdl(quantize_rows_kernel<F, BF, LAY>, dim3(grid), dim3(256), 0, st, xp, nchunks, cp, scales, S, nbd))
  if (layout == RK_SCALES_ROWMAJOR) { if (bf16) { RK_QX(true, 0); } else { RK_QX(false, 0); } }
  else if (layout == RK_SCALES_GROUPMAJOR) { if (bf16) { RK_QX(true, 1); } else { RK_QX(false, 1); } }
  else if (layout == RK_SCALES_SF_ATOMS) { if (bf16) { RK_QX(true, 2); } else { RK_QX(false, 2); } }
  else return RK_ERR_BAD_FORMAT;
#undef RK_QX
  return (int)cudaGetLastError();
}

int launch_quantize_keys_atoms(const float* x, int64_t batch, int64_t rows, int64_t cols, int fmt, uint8_t* codes,
                               uint8_t* scales, cudaStream_t st) {
  const int64_t units = batch * ((rows + 31) / 32) * ((cols + 31) / 32);
  if (units == 0) return RK_OK;
  const int grid = grid_for(units * 32, 128, 16);
  RK_DISPATCH_FMT(fmt, return (int)launch_pdl(quantize_keys_kernel<F, true>, dim3(grid), dim3(128), 0, st, x, batch, rows, cols, codes, scales));
  return RK_OK;
}

// CTAs of `threads` threads for the re-tiling jobs beside other work
static int retile_ctas(const RetileJobs& jobs, int threads) {
  int64_t atoms = 0;
  for (int i = 0; i < jobs.n; ++i) atoms += retile_atoms(jobs.job[i]);
  return atoms == 0 ? 0 : grid_for(atoms * 32, threads, 4);      // a warp each
}

int launch_retile_scales(RetileJobs jobs, cudaStream_t st) {
  if ((jobs.ctas = retile_ctas(jobs, 128)) == 0) return RK_OK;
  return (int)launch_pdl(retile_scales_kernel, dim3(jobs.ctas), dim3(128), 0, st, jobs);
}

int launch_import_kt_blocks(const uint8_t* kt, const uint8_t* kts, int64_t heads, int nblk, int Bk, int d, uint8_t* k,
                            uint8_t* ks, cudaStream_t st) {
  const int64_t ntiles = heads * nblk * (d / 32) * (Bk / 32);
  if (ntiles == 0) return RK_OK;
  import_kt_blocks_kernel<<<(int)min(ntiles, (int64_t)num_sms() * 16), 256, 0, st>>>(kt, kts, heads, nblk, Bk, d, k, ks);
  return (int)cudaGetLastError();
}

// Which kernel a call takes; `wide`: x and gamma lie on 16-byte boundaries.
// Rows by bulk copy: from a chain long enough to pay for the ring (us, staged through registers and so, one call behind another on the same buffers: 4096 bf16
// columns, 8192 rows 36.5 31.8, one 17.1 15.5; 12288 columns, 1500 rows 64.7 51.7; 2048 columns, 1 and 64 rows 9.0 9.2, 300 10.9 10.2, 4096 15.5 14.1, 16384 37.4
// 34.2; 1536 columns, 64 7.4 7.6, 300 8.7 8.3, 4096 12.3 11.6; 1024 columns, 64 5.8 6.0, 300 6.6 6.5, 4096 9.3 9.2, 9000 12.3 11.5; 512 columns 2-9 % slower
// throughout), and not for fp32, whose 134 MB of 8192 x 4096 come from HBM twice either way (55.0 56.4; one row 17.4 20.3).
static int rmsnorm_form(int64_t rows, int K, bool bf16, bool wide, int64_t sms, rms_seg::Shape& f) {
  if (g_rmsnorm_form == kRmsnormStaged || (g_rmsnorm_form == kRmsnormRing && wide && bf16)) return g_rmsnorm_form;
  if (wide && rms_seg::pays(rows, K, bf16, sms, f)) return kRmsnormSegments;
  return wide && bf16 && (K >= 2048 || (K >= 1024 && rows >= 4096)) ? kRmsnormRing : kRmsnormStaged;
}
int rmsnorm_form(int64_t rows, int K, bool bf16, int64_t sms) { rms_seg::Shape f; return rmsnorm_form(rows, K, bf16, true, sms, f); }

int launch_rmsnorm_quantize(const void* x, bool bf16, int64_t rows, int K, const float* gamma, float eps, int fmt,
                            bool unit_scale, uint8_t* codes, uint8_t* scales, cudaStream_t st) {
  if (rows == 0 || K == 0) return RK_OK;
  const bool wide = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gamma)) & 15) == 0;
  rms_seg::Shape f;
  const int form = rmsnorm_form(rows, K, bf16, wide, num_sms(), f);
  if (form == kRmsnormSegments) {
    int* status = device_status_word();
    if (!status) return RK_ERR_NO_DEVICE;
#define RK_RN(BF, UN) RK_DISPATCH_FMT(fmt, {                                                                                \
    auto kern = F == RK_FMT_E4M3 && BF && !UN && g_ring_stop ? rmsnorm_quantize_segments_kernel<RK_FMT_E4M3, true, false, true> : rmsnorm_quantize_segments_kernel<F, BF, UN, false>; \
    if (f.smem + rms_seg::kStatic > 48 * 1024) {                                                                           \
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, rms_seg::kSmem - rms_seg::kStatic); \
      if (e != cudaSuccess) return (int)e;                                                                                 \
    }                                                                                                                      \
    return (int)launch_pdl(kern, dim3((unsigned)f.grid), dim3(rms_seg::kThreads), (size_t)f.smem, st, reinterpret_cast<const uint8_t*>(x), rows, K, f.rows, f.seg, f.warps, f.pitch, gamma, eps, codes, scales, status, g_ring_stop); \
  })
    if (bf16) { if (unit_scale) { RK_RN(true, true); } else { RK_RN(true, false); } }
    else      { if (unit_scale) { RK_RN(false, true); } else { RK_RN(false, false); } }
#undef RK_RN
  }
  if (form == kRmsnormRing) {
    int* status = device_status_word();
    if (!status) return RK_ERR_NO_DEVICE;
    const int64_t slots = (int64_t)num_sms() * rmb::kCtasPerSm, waves = (rows + slots * rmb::kMaxRows - 1) / (slots * rmb::kMaxRows);
    const int per_cta = (int)((rows + slots * waves - 1) / (slots * waves));
    const int64_t grid = (rows + per_cta - 1) / per_cta;
    if (grid > 0x7FFFFFFF) return RK_ERR_BAD_SHAPE;
    const int smem = rmb::kStages * per_cta * rmb::kPitch;
#define RK_RN(UN) RK_DISPATCH_FMT(fmt, {                                                                                \
    auto kern = F == RK_FMT_E4M3 && !UN && g_ring_stop ? rmsnorm_quantize_bulk_kernel<RK_FMT_E4M3, false, true> : rmsnorm_quantize_bulk_kernel<F, UN, false>; \
    if (smem > 48 * 1024) {                                                                                                \
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, rmb::kStages * rmb::kMaxRows * rmb::kPitch); \
      if (e != cudaSuccess) return (int)e;                                                                                 \
    }                                                                                                                      \
    return (int)launch_pdl(kern, dim3((unsigned)grid), dim3(rmb::kThreads), smem, st, reinterpret_cast<const uint8_t*>(x), rows, K, per_cta, gamma, eps, codes, scales, status, g_ring_stop); \
  })
    if (unit_scale) { RK_RN(true); } else { RK_RN(false); }
#undef RK_RN
  }
  // Rows per CTA: as few whole waves of resident CTAs as kMaxRows each allow, with the rows spread evenly over them (one
  // wave and 14 rows for 8192); one row per CTA below one CTA per slot, so that few rows still reach every SM.
  const int64_t slots = (int64_t)num_sms() * rms::kCtasPerSm;
  const int64_t waves = (rows + slots * rms::kMaxRows - 1) / (slots * rms::kMaxRows);
  const int per_cta = (int)((rows + slots * waves - 1) / (slots * waves));
  const int64_t grid = (rows + per_cta - 1) / per_cta;
  if (grid > 0x7FFFFFFF) return RK_ERR_BAD_SHAPE;
  const int smem = rms::kBufs * per_cta * rms::kPitch;
  const uint8_t* xb = reinterpret_cast<const uint8_t*>(x);
#define RK_RN(BF, UN, PC) RK_DISPATCH_FMT(fmt, {                                                                            \
    auto kern = rmsnorm_quantize_kernel<F, BF, UN, PC>;                                                                    \
    if (smem > 48 * 1024) {                                                                                                \
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, rms::kBufs * rms::kMaxRows * rms::kPitch); \
      if (e != cudaSuccess) return (int)e;                                                                                 \
    }                                                                                                                      \
    return (int)launch_pdl(kern, dim3((unsigned)grid), dim3(rms::kThreads), smem, st, xb, rows, K, per_cta, gamma, eps, codes, scales); \
  })
#define RK_RNB(BF, UN) if (wide) { RK_RN(BF, UN, 16); } else { RK_RN(BF, UN, 4); }
  if (bf16) { if (unit_scale) { RK_RNB(true, true); } else { RK_RNB(true, false); } }
  else      { if (unit_scale) { RK_RNB(false, true); } else { RK_RNB(false, false); } }
#undef RK_RNB
#undef RK_RN
  return RK_OK;
}

int launch_quantize_rows(const float* x, int64_t rows, int64_t cols, int fmt, uint8_t* codes, uint8_t* scales,
                         cudaStream_t st) {
  const int64_t nchunks = rows * cols / 8;
  if (nchunks == 0) return RK_OK;
  const int grid = grid_for(nchunks, 256, 8);
  RK_DISPATCH_FMT(fmt, return (int)launch_pdl(quantize_rows_kernel<F, false, 0>, dim3(grid), dim3(256), 0, st, reinterpret_cast<const float4*>(x),
                                              nchunks, reinterpret_cast<uint2*>(codes), scales, (int64_t)0, 0));
  return RK_OK;
}

int launch_quantize_keys(const float* x, int64_t batch, int64_t rows, int64_t cols, int fmt, uint8_t* codes,
                         uint8_t* scales, cudaStream_t st) {
  const int64_t units = batch * ((rows + 31) / 32) * ((cols + 31) / 32);
  if (units == 0) return RK_OK;
  const int grid = grid_for(units * 32, 128, 16);
  RK_DISPATCH_FMT(fmt, return (int)launch_pdl(quantize_keys_kernel<F, false>, dim3(grid), dim3(128), 0, st, x, batch, rows, cols, codes, scales));
  return RK_OK;
}

// By bulk copies from where there are several tiles for each of two rounds of CTAs, and rows enough to share the caches (by chunks per SM, us, rows in
// registers and so: 1 771 4.8 5.2, 3 542 8.3 7.2, 7 085 14.5 11.8, 14 170 28.9 27.8, 28 340 57.2 52.3, one call behind another on the same buffers; with nothing
// of them in L2 the two are equal, 22.5 us and 36.9 at 7 085 and 14 170.  Eight copies: 3 542 8.3 7.4, 7 085 15.1 12.2, 14 170 28.1 29.4).
// A CTA's tile is a range of positions of one sequence, and the threads of the rows that the last one lacks are idle, which shows least where HBM sets the
// pace.  130 shapes, this kernel's time over the other's by how full the tiles are: from 7 000 chunks per SM on 0.72-1.0 0.74-0.98, 0.62-0.71 0.91-1.07, 0.53-0.56
// 1.03-1.17; below that 0.9-1.0 0.82-0.97, 0.75-0.9 0.95-1.11, sequences of 8, 4 and 1 rows in tiles of 16 1.08, 1.7 and 5.8.
bool rope_by_copies(int64_t rows, int d, int64_t seq_len, int64_t sms) {
  const int64_t copies = rows / seq_len, per_tile = ropec::kTileBytes / (d * 4), chunks = rows * (d / 16);
  if (copies < 16 || copies > 65535 || rows % seq_len != 0 || per_tile == 0 || chunks < sms * 3000) return false;
  return 100 * seq_len >= (chunks < sms * 7000 ? 90 : 72) * ((seq_len + per_tile - 1) / per_tile * per_tile);
}

int launch_rope_quantize_rows(const float* x, int64_t rows, int d, const int32_t* pos, int seq_len, int pos0, const float* cos_h,
                              const float* sin_h, int fmt, uint8_t* codes, uint8_t* scales, cudaStream_t st) {
  const int64_t nchunks = rows * (d / 16);
  if (nchunks == 0) return RK_OK;
  if (!pos && rope_by_copies(rows, d, seq_len, num_sms()) && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    const int64_t copies = rows / seq_len;
    const int per_tile = ropec::kTileBytes / (d * 4);
    int* status = device_status_word();
    if (!status) return RK_ERR_NO_DEVICE;
    const int64_t ctas = (seq_len + per_tile - 1) / per_tile, slots = 2 * (int64_t)num_sms() * ropec::kCtasPerSm;
    const dim3 grid((unsigned)ctas, (unsigned)std::min<int64_t>(std::max<int64_t>(1, slots / ctas), copies));
    RK_DISPATCH_FMT(fmt, return (int)launch_pdl(F == RK_FMT_E4M3 && g_ring_stop ? rope_quantize_copies_kernel<RK_FMT_E4M3, true> : rope_quantize_copies_kernel<F, false>, grid, dim3(ropec::kThreads), 0, st, x, (int)copies, d, seq_len, pos0, cos_h, sin_h, codes, scales, status));
  }
  // two rows per thread where every position has at least two and halving the threads still leaves every SM full
  const bool two = !pos && rows % seq_len == 0 && rows / seq_len >= 2 && nchunks >= (int64_t)num_sms() * 4096;
  // one wave of the CTAs that fit an SM, so that all end together (52 us against 49 for the Q, K, V of 8192 tokens with four)
  const dim3 grid(grid_for(two ? (nchunks + 1) / 2 : nchunks, 128, two ? 4 : 7)), block(128);
  if (two) { RK_DISPATCH_FMT(fmt, return (int)launch_pdl(rope_quantize_rows_kernel<F, 2>, grid, block, 0, st, x, rows, d, pos, seq_len, pos0, cos_h, sin_h, codes, scales)); }
  else     { RK_DISPATCH_FMT(fmt, return (int)launch_pdl(rope_quantize_rows_kernel<F, 1>, grid, block, 0, st, x, rows, d, pos, seq_len, pos0, cos_h, sin_h, codes, scales)); }
  return RK_OK;
}

int launch_kv_append(const float* k_new, const float* v_new, int B, int H_kv, int L, int d, const int32_t* pos, int fmt,
                     uint8_t* k_codes, uint8_t* k_scales, uint8_t* v_codes, uint8_t* v_scales, cudaStream_t st) {
  const int64_t chunks = (int64_t)B * H_kv * (d / 8);                   // below 2^32: 64 bytes of k_new and v_new each
  if (chunks == 0) return RK_OK;
  RK_DISPATCH_FMT(fmt, return (int)launch_pdl(kv_append_kernel<F>, dim3(grid_for(chunks, 128, 4), 2), dim3(128), 0, st, k_new, v_new, (uint32_t)(B * (int64_t)H_kv), (uint32_t)H_kv, L, (uint32_t)d, pos, k_codes, k_scales, v_codes, v_scales));
  return (int)cudaGetLastError();
}

int launch_rebase_v(const uint8_t* codes, const uint8_t* scales, int64_t batch, int64_t S, int64_t d, int fmt,
                    uint8_t* out_codes, uint8_t* out_scales, bool tiled, cudaStream_t st, RetileJobs jobs) {
  const bool small = d <= INT_MAX / 32;                  // 32 rows can be indexed by an int
  const bool wide = small && ((reinterpret_cast<uintptr_t>(codes) | reinterpret_cast<uintptr_t>(out_codes)) & 7) == 0;
  const int64_t units = batch * ((S + 127) / 128) * (wide ? (d + 63) / 64 : d / 32);
  if (units == 0) return RK_OK;
  jobs.ctas = retile_ctas(jobs, kRebaseThreads);
  const dim3 grid(jobs.ctas + grid_for(units * kRebaseThreads, kRebaseThreads, 28)), block(kRebaseThreads);      // four waves of the resident CTAs
#define RK_RB(TI, N, IDX) RK_DISPATCH_FMT(fmt, return (int)launch_pdl(rebase_v_kernel<F, TI, N, IDX>, grid, block, 0, st, codes, scales, batch, S, d, out_codes, out_scales, jobs))
  if (wide) { if (tiled) { RK_RB(true, 8, int); } else { RK_RB(false, 8, int); } }
  else if (tiled) return RK_ERR_MISALIGNED;              // (prefill's codes and workspace lie on 16-byte boundaries)
  else if (small) { RK_RB(false, 4, int); }
  else { RK_RB(false, 4, int64_t); }
#undef RK_RB
  return RK_OK;
}

int launch_pack_rows(const PackJobs& packs, int64_t d, cudaStream_t st, RetileJobs jobs) {
  const int64_t dp = (d + 127) / 128 * 128;
  int64_t most = 0;
  for (int i = 0; i < packs.n; ++i) most = std::max(most, packs.job[i].rows * (dp / 16));
  if (most == 0) return RK_OK;
  jobs.ctas = retile_ctas(jobs, 256);
  return (int)launch_pdl(pack_rows_kernel, dim3(jobs.ctas + grid_for((most + 3) / 4, 256, 16)), dim3(256), 0, st, packs, d, dp, jobs);
}

int launch_pack_v(const uint8_t* codes, const uint8_t* scales, int64_t batch, int64_t S, int64_t d, int fmt, uint8_t* out,
                  uint8_t* atoms, cudaStream_t st) {
  const int64_t Sp = (S + 127) / 128 * 128, grid = batch * (Sp / 128) * ((d + 127) / 128);
  if (grid == 0) return RK_OK;
  if (grid > 0x7FFFFFFF) return RK_ERR_BAD_SHAPE;
  auto kern = scales ? (fmt == RK_FMT_E2M3 ? pack_v_kernel<2, true> : fmt == RK_FMT_E3M2 ? pack_v_kernel<3, true> : pack_v_kernel<4, true>)
                     : (fmt == RK_FMT_E2M1 ? pack_v_kernel<4, false> : pack_v_kernel<2, false>);
  return (int)launch_pdl(kern, dim3((unsigned)grid), dim3(128), 0, st, codes, scales, S, d, Sp, out, atoms);
}

// Runs the exhaustive encoder check for one format over all 2^32 fp32 bit patterns.
int launch_verify_encoder(int fmt, unsigned long long* mismatches, uint32_t* first_bad, cudaStream_t st) {
  const int grid = num_sms() * 8;
  RK_DISPATCH_FMT(fmt, (verify_encoder_kernel<F><<<grid, 256, 0, st>>>(0ull, 1ull << 32, mismatches, first_bad)));
  return (int)cudaGetLastError();
}

}  // namespace rk
