// Shared device helpers: MX codecs (bit-exact with the CPU oracle) and thin
// wrappers over the sm_100a PTX the kernels use (mbarrier, TMA, tcgen05/TMEM).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define RK_DEVINL __device__ __forceinline__

namespace rk {

// ----------------------------------------------------------------------------
// Element formats: {ebits, mbits, bias, unbiased emax, max mantissa, fp32
// mantissa of the largest finite value}.  Same table as the CPU oracle.
// ----------------------------------------------------------------------------
struct FmtDesc { int ebits, mbits, bias, emax, max_mant; uint32_t thresh; float fmax; };

template <int FMT> struct FmtT;
template <> struct FmtT<0> { static constexpr int ebits = 4, mbits = 3, bias = 7,  emax = 8,  max_mant = 6; static constexpr uint32_t thresh = 0x600000u; };
template <> struct FmtT<1> { static constexpr int ebits = 5, mbits = 2, bias = 15, emax = 15, max_mant = 3; static constexpr uint32_t thresh = 0x600000u; };
template <> struct FmtT<2> { static constexpr int ebits = 2, mbits = 3, bias = 1,  emax = 2,  max_mant = 7; static constexpr uint32_t thresh = 0x700000u; };
template <> struct FmtT<3> { static constexpr int ebits = 3, mbits = 2, bias = 3,  emax = 4,  max_mant = 3; static constexpr uint32_t thresh = 0x600000u; };
// E2M1 (FP4; lib/golden/mx_fp_math.h:238-246 fp4_e2m1_decode): 0, 0.5, 1, 1.5, 2, 3, 4, 6
template <> struct FmtT<4> { static constexpr int ebits = 2, mbits = 1, bias = 1,  emax = 2,  max_mant = 1; static constexpr uint32_t thresh = 0x400000u; };

template <int FMT> RK_DEVINL float fmt_max() {
  using F = FmtT<FMT>;
  // (1 + max_mant/2^mbits) * 2^emax as an fp32 bit pattern
  return __uint_as_float(((uint32_t)(F::emax + 127) << 23) | ((uint32_t)F::max_mant << (23 - F::mbits)));
}

// round-half-to-even of v >> sh (sh >= 1; sh >= 32 gives 0), the integer
// rounding of kernels/simt_quant/kernel.cpp:44-54.
RK_DEVINL uint32_t round_shift(uint32_t v, int sh) {
  if (sh >= 32) return 0u;
  const uint32_t low = v & ((1u << sh) - 1u), half = 1u << (sh - 1);
  uint32_t q = v >> sh;
  q += (low > half || (low == half && (q & 1u))) ? 1u : 0u;
  return q;
}

// fp32 -> element code, RNE, saturating; kernels/simt_quant/kernel.cpp:56-81
// generalised over the format widths.
template <int FMT> RK_DEVINL uint32_t encode_rne(float xf) {
  using F = FmtT<FMT>;
  constexpr int nb = 1 + F::ebits + F::mbits;
  constexpr uint32_t one = 1u << F::mbits;
  constexpr uint32_t sat = (uint32_t)(((F::emax + F::bias) << F::mbits) | F::max_mant);
  constexpr int emin = 1 - F::bias;
  const uint32_t x = __float_as_uint(xf);
  const uint32_t absx = x & 0x7FFFFFFFu;
  const uint32_t s = (x >> 31) << (nb - 1);
  if (absx == 0u) return s;
  if (__uint_as_float(absx) >= fmt_max<FMT>()) return s | sat;
  const int e = (int)(absx >> 23) - 127;
  const uint32_t sig = (1u << 23) | (absx & 0x7FFFFFu);
  uint32_t out;
  if (e < emin) {
    const uint32_t q = round_shift(sig, (23 - F::mbits) + (emin - e));
    out = q;   // q >= one encodes the smallest normal: (1<<mbits)|(q-one) == q
  } else {
    uint32_t r = round_shift(sig, 23 - F::mbits);
    int E = e;
    if (r == 2 * one) { r = one; E += 1; }
    const int expf = E + F::bias;
    const uint32_t mant = r - one;
    constexpr int expf_max = F::emax + F::bias;
    if (expf > expf_max || (expf == expf_max && (int)mant > F::max_mant)) return s | sat;
    out = ((uint32_t)expf << F::mbits) | mant;
  }
  return s | out;
}

// Block scale of the lib/golden rule from the fp32 bits of amax (amax > 0):
// e = ceil(log2(amax / FMT_MAX)); returns e, the clamped E8M0 code and 2^-e.
template <int FMT> RK_DEVINL void block_scale(float amax, uint32_t& code, float& pow2_neg_e) {
  using F = FmtT<FMT>;
  // the carry of the addition is the "+1 above the largest mantissa"; t = biased exponent of amax with it
  const uint32_t t = (__float_as_uint(amax) + (0x7FFFFFu - F::thresh)) >> 23;
  code = (uint32_t)max((int)t - F::emax, 0);                            // at most 255 - emax
  pow2_neg_e = __uint_as_float((uint32_t)(254 + F::emax - (int)t) << 23);
}

// Exact decode of an element code to fp32.
template <int FMT> RK_DEVINL float decode_elem(uint32_t code) {
  using F = FmtT<FMT>;
  constexpr int nb = 1 + F::ebits + F::mbits;
  const uint32_t s = (code >> (nb - 1)) & 1u;
  const uint32_t e = (code >> F::mbits) & ((1u << F::ebits) - 1u);
  const uint32_t m = code & ((1u << F::mbits) - 1u);
  float v;
  if (e == 0) v = (float)m * __uint_as_float((uint32_t)(127 + 1 - F::bias - F::mbits) << 23);
  else v = __uint_as_float(((e + 127 - F::bias) << 23) | (m << (23 - F::mbits)));
  return s ? -v : v;
}

// E8M0 -> fp32 (code 0 = 2^-127 is an fp32 denormal; 0xFF must not be passed).
RK_DEVINL float e8m0_to_f32(uint32_t c) { return __uint_as_float(c == 0 ? 0x00400000u : (c << 23)); }

// Offset of (row r of a 128-row tile, 32-element block kb of a 128-element
// chunk) inside a 512-byte scale-factor atom: 32 rows x 16 bytes, row r%32,
// byte (r/32)*4 + kb.  One tcgen05.cp 32x128b.warpx4 moves an atom to 4 TMEM
// columns (lane = r%32, column = r/32, byte = kb).
__host__ __device__ inline int sf_atom_offset(int r, int kb) { return (r & 31) * 16 + (r >> 5) * 4 + kb; }

// ----------------------------------------------------------------------------
// PTX wrappers
// ----------------------------------------------------------------------------
RK_DEVINL uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// The first 1024-byte boundary of a dynamic shared array.  By an offset: after a cast through an integer the compiler no longer knows
// that the pointer is into shared memory, stores become generic ones and every address it keeps takes two registers (d = 256
// prefill, capped, 16 heads of 8192: 1065 us with the cast, 1017 without; 509 queries behind 3581 keys 47.2 -> 46.4).  The decode
// kernels keep the cast: the mma.sync kernel is 6-10 % faster with it (other registers, other order), the tcgen05 kernel within 2 % either way.
RK_DEVINL uint8_t* align_smem(uint8_t* p) { return p + ((0u - smem_u32(p)) & 1023u); }

RK_DEVINL void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
RK_DEVINL void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
RK_DEVINL void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// One poll of an mbarrier phase.  HINT_NS > 0 lets the hardware keep the thread suspended for up to that many
// ns before it reports "not yet": a warp that waits long (a TMA producer) then issues few instructions and
// leaves the issue slots of its scheduler to the working warps; 0 = the hardware default, quickest wake-up.
template <uint32_t HINT_NS = 0>
RK_DEVINL bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  if (HINT_NS > 0) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(HINT_NS) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  }
  return ok != 0;
}
// Non-blocking test of an mbarrier phase (never suspends the thread): for a look ahead whose answer is used later.
RK_DEVINL bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
RK_DEVINL uint64_t global_timer_ns() {
  uint64_t t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t;
}
// Bounded wait: gives up after about `limit_ns` of wall time (or as soon as this
// CTA's abort flag or the device status word is set by someone else), records
// `code` in *status and returns false; the caller then skips its work so the
// kernel drains and exits instead of hanging the GPU.
// (Measured: a tighter five-instruction polling loop is slower, prefill -8 %, decode -6 %; a nanosleep of
// 20-400 ns between polls changes nothing.)
template <uint32_t HINT_NS = 0>
RK_DEVINL bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code,
                         uint64_t limit_ns = 2000000000ull) {
  if (mbar_try_wait<HINT_NS>(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait<HINT_NS>(bar, parity)) return true;
    if ((it & 255u) == 0u) {
      if (*abort_flag || *reinterpret_cast<volatile int*>(status) != 0) { *abort_flag = 1; return false; }
      if (global_timer_ns() - t0 > limit_ns) break;
    }
  }
  *abort_flag = 1;
  atomicCAS(status, 0, code);
  return false;
}

// The same bound in a form that costs a dozen instructions where it is inlined: SM cycles instead of the global
// timer, and nothing recorded here.  The caller reports the failure (report_wait_failure) outside its hot loop.
constexpr long long kWaitLimitCycles = 4000000000ll;      // about two seconds at 1.9 GHz
RK_DEVINL bool mbar_wait_lean(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait<0>(bar, parity)) return true;
  const long long t0 = clock64();
  do {
    if (mbar_try_wait<0>(bar, parity)) return true;
  } while (!*abort_flag && clock64() - t0 < kWaitLimitCycles);
  return false;
}
// The same in a dozen instructions: for kernels whose code competes for the instruction cache.  LONG: a wait off the critical path; the
// hardware may hold the warp for 2 us before it polls again, which leaves the issue slots to the others (a short prefill on 128 SMs
// 45.8 -> 44.5 us; on the softmax warps' own waits it costs 2 %).
// The caller keeps the code of the wait that gave up and reports it once, outside its loops.  abort_flag nullptr: waits on when the
// CTA has given up (drains).
template <bool LONG = false>
RK_DEVINL bool mbar_wait_short(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t t0 = (uint32_t)clock();
#pragma unroll 1
  while (!mbar_try_wait<LONG ? 2000 : 0>(bar, parity))
    if ((abort_flag && *abort_flag) || (uint32_t)clock() - t0 > (uint32_t)kWaitLimitCycles) return false;
  return true;
}
constexpr uint32_t kPollsLong = 1u << 20, kPollsShort = 1u << 22;
// The same in nine instructions, without a clock: bounded by the number of polls, which the hardware may hold for 2 us (LONG) and 0.5 us each, and does: with an
// idle SM either form runs out after 2.15 s.  (A poll may come back sooner; the limit is then shorter, 2^20 or 2^22 polls of some 40 cycles at least.)  A kernel whose warps are in different
// code all the time lives by the size of that code (an SM's instruction cache holds 32 KB): one query tile per CTA, d <= 128, 166 K instruction requests to the
// next cache level in 38.9 us, 61 % of what it can serve.  With these waits there 73.3 -> 66.8 KB of code and 36.8 -> 35.6 us, 8 heads of 4096 42.3 -> 40.2.  In
// all warps but the softmax's of pairs of query tiles, 2 x 16 heads of 4096 137.7 -> 134.1 us, 32 / 8 of 8192 455 -> 448 (in the softmax warps as well: 467).
// Not at d = 256, whose long sequences lose: 16 / 8 heads of 8192 with a cap 957 -> 966, whichever of its warps wait so.
template <bool LONG = false, uint32_t POLLS = LONG ? kPollsLong : kPollsShort>
RK_DEVINL bool mbar_wait_compact(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 n, f;\n\t"
      "mov.u32 n, %4;\n\t"
      "POLL_%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "@p bra OVER_%=;\n\t"
      "ld.volatile.shared.u32 f, [%5];\n\t"
      "setp.ne.u32 q, f, 0;\n\t"
      "@q bra OVER_%=;\n\t"
      "sub.u32 n, n, 1;\n\t"
      "setp.ne.u32 q, n, 0;\n\t"
      "@q bra POLL_%=;\n\t"
      "OVER_%=:\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "n"(LONG ? 2000 : 500), "n"(POLLS), "r"(smem_u32(const_cast<int*>(abort_flag))) : "memory");
  return ok != 0;
}
RK_DEVINL void report_wait_failure(volatile int* abort_flag, int* status, int code) {
  *abort_flag = 1;
  atomicCAS(status, 0, code);
}

// Programmatic dependent launch: a kernel launched with the attribute starts while the one before it in the stream still
// runs; it waits here before it touches anything that one may write (or read, where it writes), and lets the one after
// it start.  Both do nothing in an ordinary launch.
RK_DEVINL void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
RK_DEVINL void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

RK_DEVINL void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
RK_DEVINL void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// TMA: 3-D tiled load global -> shared, completion on an mbarrier.
RK_DEVINL void tma_load_3d(void* smem_dst, const void* tmap, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
// TMA: 1-D bulk copy global -> shared (16-byte aligned, size multiple of 16).
RK_DEVINL void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// TMA: 3-D tiled store shared -> global (what lies outside the tensor is left out); completion by bulk groups.
RK_DEVINL void tma_store_3d(const void* tmap, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(tmap), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z) : "memory");
}
RK_DEVINL void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> RK_DEVINL void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }   // at most N groups still read their source
RK_DEVINL void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
RK_DEVINL void prefetch_tmap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// Cluster launch control: a running CTA takes over the block index of one that has not started yet.  The answer (16 bytes) arrives
// in shared memory and completes 16 bytes on the mbarrier.  After an answer "none left" no further request may be made.
RK_DEVINL void clc_request(void* smem_answer, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(smem_answer)), "r"(smem_u32(bar)) : "memory");
}
RK_DEVINL bool clc_answer(const void* smem_answer, uint32_t& block_x) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .b128 r;\n\t.reg .b64 lo, hi;\n\t.reg .pred p;\n\t"
      "ld.shared.v2.b64 {lo, hi}, [%2];\n\t"
      "mov.b128 r, {lo, hi};\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
      : "=r"(ok), "=r"(block_x) : "r"(smem_u32(smem_answer)) : "memory");
  return ok != 0;
}

// One lane of a converged warp, the same one every time.
RK_DEVINL bool elect_one() {
  uint32_t is;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(is));
  return is != 0;
}
// A value that is the same in all lanes, in a form the compiler knows to be.
RK_DEVINL int warp_uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }

// ---- TMEM / tcgen05 ----
RK_DEVINL void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {   // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
RK_DEVINL void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
RK_DEVINL void tmem_dealloc(uint32_t taddr, uint32_t ncols) {     // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
RK_DEVINL void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
RK_DEVINL void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
RK_DEVINL void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
RK_DEVINL void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// mbarrier arrives once every tcgen05 op issued so far by this thread is done.
RK_DEVINL void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Block-scaled MMA, operands in shared memory, E8M0 scales in TMEM:
// D[tmem] (+)= (A * sfa) . (B * sfb), one 32-deep K slice.
RK_DEVINL void mma_mxf8f6f4_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                               uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem) : "memory");
}
// 32 rows x 16 bytes of shared memory -> 4 TMEM columns, replicated into all
// four 32-lane quadrants (the scale-factor copy).
RK_DEVINL void tc_cp_32x128b_warpx4(uint32_t dst_tmem, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(dst_tmem), "l"(sdesc) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets lane
// (base lane + i), registers r[0..31] = columns taddr.col + 0..31.
RK_DEVINL void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
RK_DEVINL void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
RK_DEVINL void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
RK_DEVINL void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
RK_DEVINL void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
RK_DEVINL void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// Shared-memory matrix descriptor (sm_100 format): start address, leading and
// stride byte offsets in 16-byte units, descriptor version 1 at bits 46-47,
// layout type at bits 61-63 (0 = no swizzle, 2 = 128-byte swizzle).
RK_DEVINL uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)(layout & 7u) << 61;
  return d;
}
constexpr uint32_t kLayoutNone = 0, kLayoutSw128 = 2;

// Instruction descriptor of kind::mxf8f6f4.block_scale (dense):
//  [4,6) B scale id  [7,10) A format  [10,13) B format  [15] A MN-major  [16] B MN-major
//  [17,23) N>>3  [23] scale format (1 = E8M0)  [24,29) M>>4  [29,31) A scale id
// Hardware element-format ids: E4M3 0, E5M2 1, E2M3 3, E3M2 4, E2M1 5.
__host__ __device__ inline constexpr uint32_t hw_fmt_id(int fmt) { return fmt == 0 ? 0u : fmt == 1 ? 1u : fmt == 2 ? 3u : fmt == 3 ? 4u : 5u; }
__host__ __device__ inline constexpr uint32_t make_idesc(int a_fmt, int b_fmt, bool a_mn, bool b_mn, int M, int N) {
  return (hw_fmt_id(a_fmt) << 7) | (hw_fmt_id(b_fmt) << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(N >> 3) << 17) | (1u << 23) | ((uint32_t)(M >> 4) << 24);
}
RK_DEVINL uint32_t idesc_with_sf(uint32_t idesc, uint32_t a_sf_id, uint32_t b_sf_id) {
  return idesc | (b_sf_id << 4) | (a_sf_id << 29);
}

RK_DEVINL float ex2_approx(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
RK_DEVINL float rcp_approx(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

}  // namespace rk
