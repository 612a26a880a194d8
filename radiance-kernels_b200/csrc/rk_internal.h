// Declarations shared by the .cu files of the library (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rk_mx_attn.h"

namespace rk {

extern cudaEvent_t g_ev_before, g_ev_after;   // optional profiling events around the main kernels
int num_sms();                 // SM count of the current device (cached per device)
int* device_status_word();     // per-device int inside the library image, zero at load; kernels CAS error codes into it.
                               // NULL when the device could not be queried: callers return RK_ERR_NO_DEVICE

int launch_quantize_rows_bf16(const void* x, int64_t rows, int64_t cols, int fmt, uint8_t* codes, uint8_t* scales, cudaStream_t st);
int launch_quantize_rows(const float* x, int64_t rows, int64_t cols, int fmt, uint8_t* codes, uint8_t* scales, cudaStream_t st);
int launch_quantize_keys(const float* x, int64_t batch, int64_t rows, int64_t cols, int fmt, uint8_t* codes, uint8_t* scales, cudaStream_t st);
// Block scales to re-tile into scale-factor atoms beside other preparation work: up to Q's, K's and V's (kind: where they lie,
// see retile_scales_body).
struct RetileJob { const uint8_t* in; uint8_t* out; int64_t batch, S, d; int kind; };
struct RetileJobs { int n, ctas; RetileJob job[3]; };      // ctas: set by the launch functions
int launch_rebase_v(const uint8_t* codes, const uint8_t* scales, int64_t batch, int64_t S, int64_t d, int fmt,
                    uint8_t* out_codes, uint8_t* out_scales, bool tiled, cudaStream_t st, RetileJobs jobs);
int launch_retile_scales(RetileJobs jobs, cudaStream_t st);
struct PackJob { const uint8_t* in; uint8_t* out; int64_t rows; int bits; };     // byte codes [rows][d] -> dense rows
struct PackJobs { int n; PackJob job[2]; };
int launch_pack_rows(const PackJobs& packs, int64_t d, cudaStream_t st, RetileJobs jobs);
// V [batch][S][d], one code per byte -> dense transposed [batch][d][Sp * bits / 8].  scales != nullptr: V is scaled along d and is
// re-blocked along the keys on the way, the new scales going to `atoms`.
int launch_pack_v(const uint8_t* codes, const uint8_t* scales, int64_t batch, int64_t S, int64_t d, int fmt, uint8_t* out,
                  uint8_t* atoms, cudaStream_t st);
int launch_verify_encoder(int fmt, unsigned long long* mismatches, uint32_t* first_bad, cudaStream_t st);
int launch_quantize_rows_ex(const void* x, bool bf16, int64_t batch, int64_t S, int64_t d, int fmt, uint8_t* codes,
                            uint8_t* scales, int layout, cudaStream_t st);
int launch_quantize_keys_atoms(const float* x, int64_t batch, int64_t rows, int64_t cols, int fmt, uint8_t* codes,
                               uint8_t* scales, cudaStream_t st);
int launch_rmsnorm_quantize(const void* x, bool bf16, int64_t rows, int K, const float* gamma, float eps, int fmt,
                            bool unit_scale, uint8_t* codes, uint8_t* scales, cudaStream_t st);
int launch_mx_gemm_hw(const uint8_t* A, const uint8_t* B, const uint8_t* SA, const uint8_t* SB, int M, int N, int K,
                      uint16_t* C, cudaStream_t st);
int launch_import_kt_blocks(const uint8_t* kt, const uint8_t* kts, int64_t heads, int nblk, int Bk, int d, uint8_t* k,
                            uint8_t* ks, cudaStream_t st);

// q/k/v_codes: byte codes as the caller gave them, or -- for 6- and 4-bit formats -- the packed copies made by
// launch_pack_rows (Q, K) and launch_pack_v (V, stored [d][keys]).
// prepares: the attention kernel puts the scales into atoms and re-blocks V itself (prefill_prepares); codes and scales are then the caller's.
int launch_prefill(const rk_prefill_args& a, const uint8_t* q_codes, const uint8_t* k_codes, const uint8_t* v_codes,
                   const uint8_t* q_sf, const uint8_t* k_sf, const uint8_t* v_sf, bool prepares, cudaStream_t st);
bool prefill_prepares(const rk_prefill_args& a);

// RMSNorm: rows staged through registers, by bulk copies in a ring with a chain per lane, or whole on the chip with their chains cut into segments.
enum RmsnormForm { kRmsnormStaged = 1, kRmsnormRing = 2, kRmsnormSegments = 3 };
int rmsnorm_form(int64_t rows, int K, bool bf16, int64_t sms);               // which of them a call with x and gamma on 16-byte boundaries takes
bool rope_by_copies(int64_t rows, int d, int64_t seq_len, int64_t sms);      // which RoPE kernel a call without positions of its own takes
// Which kernel a prefill call takes on a device of `sms` SMs: d = 256, pairs of query tiles, one query tile at a time with the softmax groups on alternate
// key tiles, one query tile per CTA with both groups on every key tile.
enum PrefillForm { kFormWide = 0, kFormPairs = 1, kFormTurns = 2, kFormSplit = 3 };
int prefill_form(const rk_prefill_args& a, int64_t sms);

int launch_rope_quantize_rows(const float* x, int64_t rows, int d, const int32_t* pos, int seq_len, int pos0, const float* cos_h,
                              const float* sin_h, int fmt, uint8_t* codes, uint8_t* scales, cudaStream_t st);
int launch_kv_append(const float* k_new, const float* v_new, int B, int H_kv, int L, int d, const int32_t* pos, int fmt,
                     uint8_t* k_codes, uint8_t* k_scales, uint8_t* v_codes, uint8_t* v_scales, cudaStream_t st);
int launch_decode(const rk_decode_args& a, int num_splits, cudaStream_t st);
int launch_decode_noalloc(const rk_decode_args& a, cudaStream_t st);
int noalloc_status_read_clear();                            // status word of the no-allocation decode path: read, then clear
int launch_mxfp8_mma_loop(const uint8_t* a_tile, const uint8_t* b_tile, int iters, cudaStream_t st);   // tensor-pipe ceiling probe
int launch_wait_runs_out(int limit_us, bool noalloc, cudaStream_t st);   // test hook: a bounded wait that must give up
int launch_compact_wait_runs_out(bool longer, bool aborted, cudaStream_t st);      // test hook: the same for the waits bounded by a number of polls
extern int g_ring_stop;                                     // test hook: a role of the RoPE and RMSNorm kernels' rings of copies acts as if its wait had run out
extern int g_rmsnorm_form;                                  // test hook: RmsnormForm of the next calls that can take it (staged; ring), 0 = by the rule
extern int g_decode_path;                                   // test hook: 0 = by shape, 1 = mma.sync kernel only
bool decode_uses_tc(const rk_decode_args& a);                // true when the tcgen05 decode kernel serves this call
size_t decode_workspace_bytes(const rk_decode_args& a, int num_splits);   // of the kernel that serves the call, at its full grid
size_t decode_workspace_least(const rk_decode_args& a, int num_splits);   // the smallest it runs with

// Launch with the programmatic attribute: the kernel's set-up runs while the kernel before it in the stream finishes.  Only
// for kernels in which every CTA calls grid_dependency_wait() before it touches memory another kernel may use.
template <class... P, class... A>
cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cfg.attrs = attr; cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  if (e != cudaSuccess) cudaGetLastError();      // reported here, not by the next call that asks for the last error as well
  return e;
}

}  // namespace rk
