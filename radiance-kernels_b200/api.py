"""Torch-tensor front end of the C ABI (include/rk_mx_attn.h).

Argument names and meaning follow the reference kernels' data headers
(kernels/flash_attention_mx_gemma/fa_gen_data.py:148-192): Q/K/V element codes
with E8M0 block scales, B/H/H_kv/S/d, q_pos0, causal, window, softcap,
softmax_scale.  torch is used for device memory and streams only; all math runs
in the library's CUDA kernels.
"""
import ctypes as C

import torch

from ._lib import DecodeArgs, PrefillArgs, check, front, lib

E4M3, E5M2, E2M3, E3M2, E2M1 = 0, 1, 2, 3, 4
V_SCALES_ALONG_KEYS, V_SCALES_ALONG_D = 0, 1
SCALES_ROWMAJOR, SCALES_GROUPMAJOR, SCALES_SF_ATOMS = 0, 1, 2


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _need_cuda(*ts):
    for t in ts:
        if t is not None and (not t.is_cuda or not t.is_contiguous()):
            raise ValueError("expected contiguous CUDA tensors")


def _expect(t, name, dtype, shape):
    """A wrong dtype or shape must become a ValueError here: past this point the tensor is a raw pointer that TMA
    and bulk copies read with the sizes of the argument struct."""
    if t is None:
        return
    if t.dtype != dtype:
        raise ValueError(f"{name}: expected dtype {dtype}, got {t.dtype}")
    if tuple(t.shape) != tuple(shape):
        raise ValueError(f"{name}: expected shape {tuple(shape)}, got {tuple(t.shape)}")


def _check_prefill_tensors(q, k, v, q_scale, k_scale, v_scale, o, lse, v_scale_axis, q_scale_layout=SCALES_ROWMAJOR,
                           k_scale_layout=SCALES_ROWMAJOR, v_scale_layout=SCALES_ROWMAJOR):
    front().check_prefill_tensors(q, k, v, q_scale, k_scale, v_scale, o, lse, v_scale_axis, q_scale_layout, k_scale_layout,
                                  v_scale_layout)


def mx_quantize(x, fmt=E4M3):
    """fp32 or bf16 [..., cols] -> (codes uint8 [..., cols], scales uint8 [..., cols/32]); blocks along the last axis."""
    return front().mx_quantize(x, fmt)


def mx_quantize_ex(x, fmt=E4M3, scale_layout=SCALES_ROWMAJOR):
    """fp32 or bf16 [..., S, d] -> (codes [..., S, d], scales in `scale_layout` per [S, d] matrix): row-major
    [..., S, d/32], group-major [..., d/32, S] or scale-factor atoms [..., ceil(S/128), ceil(d/128), 512]."""
    return front().mx_quantize_ex(x, fmt, scale_layout)


def mx_quantize_keys_ex(x, fmt=E4M3, scale_layout=SCALES_ROWMAJOR):
    """fp32 [..., rows, cols], blocks down the rows -> codes and scales row-major [..., ceil(rows/32), cols] or
    scale-factor atoms [..., ceil(rows/128), ceil(cols/128), 512]."""
    return front().mx_quantize_keys(x, fmt, scale_layout)


def import_kt_blocks(kt_blocks, kt_scale_blocks, heads, n_blocks, Bk, d):
    """The reference's per-block K^T tiles [heads*n_blocks*d, Bk] and group-major scales [heads*n_blocks*d/32, Bk]
    -> natural K codes [heads, n_blocks*Bk, d] and row-major scales [heads, n_blocks*Bk, d/32]."""
    _need_cuda(kt_blocks, kt_scale_blocks)
    _expect(kt_blocks, "kt_blocks", torch.uint8, (heads * n_blocks * d, Bk))
    _expect(kt_scale_blocks, "kt_scale_blocks", torch.uint8, (heads * n_blocks * (d // 32), Bk))
    k = torch.empty((heads, n_blocks * Bk, d), dtype=torch.uint8, device=kt_blocks.device)
    ks = torch.empty((heads, n_blocks * Bk, d // 32), dtype=torch.uint8, device=kt_blocks.device)
    check(lib().rk_import_kt_blocks(_ptr(kt_blocks), _ptr(kt_scale_blocks), heads, n_blocks, Bk, d, _ptr(k), _ptr(ks), _stream()),
          "rk_import_kt_blocks")
    return k, ks


def rope_mx_quantize(x, cos_half, sin_half, *, pos=None, pos0=0, fmt=E4M3):
    """RoPE (rotate-half) then MX quantization along d.  x fp32 [..., S, d]; caches fp32 [n_pos, d/2]; rows use cache
    row pos0 + s, or pos[row] (int32 tensor with one entry per row) when given.  Returns (codes, scales)."""
    return front().rope_mx_quantize(x, cos_half, sin_half, pos, pos0, fmt)


def rmsnorm_mx_quantize(x, gamma, eps, fmt=E4M3, unit_scale=False):
    """Row RMSNorm (the reference's fp32 order) then quantization along the last axis.  x fp32 or bf16 [..., K];
    gamma fp32 [K].  Returns (codes [..., K], scales [..., K/32]); unit_scale: E4M3 under 2^0, scales all 0x7F."""
    return front().rmsnorm_mx_quantize(x, gamma, eps, fmt, unit_scale)


def mx_gemm_hw(a, b, a_scales, b_scales):
    """MX matmul in the mesh's accumulate semantics (bit-exact with the reference's mx_golden program).  a [M,K], b [K,N]
    E4M3 codes; a_scales [K/32,M], b_scales [K/32,N] E8M0 codes.  Returns C as bf16 [M,N]."""
    _need_cuda(a, b, a_scales, b_scales)
    if a.dim() != 2 or b.dim() != 2:
        raise ValueError("a must be [M,K] and b [K,N]")
    M, K = a.shape
    N = b.shape[1]
    _expect(a, "a", torch.uint8, (M, K)); _expect(b, "b", torch.uint8, (K, N))
    _expect(a_scales, "a_scales", torch.uint8, (K // 32, M)); _expect(b_scales, "b_scales", torch.uint8, (K // 32, N))
    c = torch.empty((M, N), dtype=torch.bfloat16, device=a.device)
    check(lib().rk_mx_gemm_hw(_ptr(a), _ptr(b), _ptr(a_scales), _ptr(b_scales), M, N, K, _ptr(c), _stream()), "rk_mx_gemm_hw")
    return c


def mx_quantize_keys(x, fmt=E4M3):
    """fp32 [..., rows, cols] -> codes same shape, scales [..., ceil(rows/32), cols]; blocks run down the rows."""
    return front().mx_quantize_keys(x, fmt, SCALES_ROWMAJOR)


def mx_rebase_v(codes, scales, fmt=E4M3):
    """[..., S, d] codes + [..., S, d/32] scales -> codes [..., S, d] + scales [..., ceil(S/32), d] (blocks along keys)."""
    return front().mx_rebase_v(codes, scales, fmt)


def _prefill_args(q, k, v, q_scale, k_scale, v_scale, o, lse, causal, softmax_scale, q_pos0, window, softcap,
                  q_fmt, kv_fmt, v_scale_axis, q_scale_layout=SCALES_ROWMAJOR, k_scale_layout=SCALES_ROWMAJOR,
                  v_scale_layout=SCALES_ROWMAJOR):
    B, H, S_q, d = q.shape
    H_kv, S_kv = k.shape[1], k.shape[2]
    a = PrefillArgs()
    a.q, a.k, a.v = _ptr(q), _ptr(k), _ptr(v)
    a.q_scale, a.k_scale, a.v_scale = _ptr(q_scale), _ptr(k_scale), _ptr(v_scale)
    a.o, a.lse = _ptr(o), _ptr(lse)
    a.B, a.H, a.H_kv, a.S_q, a.S_kv, a.d = B, H, H_kv, S_q, S_kv, d
    a.q_pos0, a.causal, a.window = q_pos0, int(bool(causal)), window
    a.softcap, a.softmax_scale = float(softcap), float(softmax_scale)
    a.q_fmt, a.kv_fmt, a.v_scale_axis, a.block_n = q_fmt, kv_fmt, v_scale_axis, 0
    a.q_scale_layout, a.k_scale_layout, a.v_scale_layout = q_scale_layout, k_scale_layout, v_scale_layout
    return a


def attn_prefill_workspace_bytes(B, H, H_kv, S_q, S_kv, d, v_scale_axis=V_SCALES_ALONG_D, q_fmt=E4M3, kv_fmt=E4M3):
    a = PrefillArgs()
    a.B, a.H, a.H_kv, a.S_q, a.S_kv, a.d = B, H, H_kv, S_q, S_kv, d
    a.v_scale_axis, a.q_fmt, a.kv_fmt = v_scale_axis, q_fmt, kv_fmt
    return lib().rk_attn_prefill_workspace_bytes(C.byref(a))


def attn_prefill(q, k, v, q_scale, k_scale, v_scale, *, causal, softmax_scale=0.0, q_pos0=0, window=0, softcap=0.0,
                 q_fmt=E4M3, kv_fmt=E4M3, v_scale_axis=V_SCALES_ALONG_D, q_scale_layout=SCALES_ROWMAJOR,
                 k_scale_layout=SCALES_ROWMAJOR, v_scale_layout=SCALES_ROWMAJOR, out=None, lse=None, workspace=None):
    """MX flash-attention prefill.  q [B,H,S_q,d], k/v [B,H_kv,S_kv,d] uint8 codes; scales as the C header says.
    Returns O bf16 [B,H,S_q,d]."""
    return front().attn_prefill(q, k, v, q_scale, k_scale, v_scale, out, lse, workspace, v_scale_axis, causal, softmax_scale,
                                q_pos0, window, softcap, q_fmt, kv_fmt, q_scale_layout, k_scale_layout, v_scale_layout)


def mx_pack_rows(codes, fmt):
    """6- or 4-bit codes one per byte [..., d] -> the dense rows form [..., dp * bits / 8] (dp = d rounded up to 128)."""
    _need_cuda(codes)
    if codes.dtype != torch.uint8 or codes.dim() < 2:
        raise ValueError("mx_pack_rows takes uint8 codes [..., d]")
    d = codes.shape[-1]
    rows = codes.numel() // max(d, 1)
    nbytes = lib().rk_mx_packed_rows_bytes(rows, d, fmt)
    if nbytes == 0 and rows > 0:
        raise ValueError("mx_pack_rows: format has no dense form (E2M3, E3M2, E2M1 only)")
    out = torch.empty(codes.shape[:-1] + (nbytes // max(rows, 1),), dtype=torch.uint8, device=codes.device)
    check(lib().rk_mx_pack_rows(_ptr(codes), rows, d, fmt, _ptr(out), _stream()), "rk_mx_pack_rows")
    return out


def mx_pack_vt(v_codes, fmt):
    """V codes blocked along the keys, one per byte [..., S, d] -> the dense transposed form [..., d, Sp * bits / 8]."""
    _need_cuda(v_codes)
    if v_codes.dtype != torch.uint8 or v_codes.dim() < 2:
        raise ValueError("mx_pack_vt takes uint8 codes [..., S, d]")
    S, d = v_codes.shape[-2], v_codes.shape[-1]
    batch = v_codes.numel() // max(S * d, 1)
    nbytes = lib().rk_mx_packed_vt_bytes(batch, S, d, fmt)
    if nbytes == 0 and batch > 0:
        raise ValueError("mx_pack_vt: format has no dense form (E2M3, E3M2, E2M1 only)")
    out = torch.empty(v_codes.shape[:-2] + (d, nbytes // max(batch * d, 1)), dtype=torch.uint8, device=v_codes.device)
    check(lib().rk_mx_pack_vt(_ptr(v_codes), batch, S, d, fmt, _ptr(out), _stream()), "rk_mx_pack_vt")
    return out


def attn_prefill_packed(q, k, vt, q_scale, k_scale, v_scale, *, S_q, S_kv, d, q_fmt, kv_fmt, causal, softmax_scale=0.0,
                        q_pos0=0, window=0, softcap=0.0, q_scale_layout=SCALES_ROWMAJOR, k_scale_layout=SCALES_ROWMAJOR,
                        v_scale_layout=SCALES_ROWMAJOR, out=None, lse=None, workspace=None):
    """Prefill over dense 6- / 4-bit operands: q [B,H,S_q,*] and k [B,H_kv,S_kv,*] from mx_pack_rows, vt
    [B,H_kv,d,*] from mx_pack_vt (V blocked along the keys, v_scale along the keys).  Returns O bf16 [B,H,S_q,d]."""
    return front().attn_prefill_packed(q, k, vt, q_scale, k_scale, v_scale, out, lse, workspace, S_q, S_kv, d, causal,
                                       softmax_scale, q_pos0, window, softcap, q_fmt, kv_fmt, q_scale_layout, k_scale_layout,
                                       v_scale_layout)


class PrefillHostRunner:
    """Prefill through the host-buffer entry point (rk_attn_prefill_host): inputs and output live in
    pinned host memory, the device arena is allocated once and reused."""

    def __init__(self, q, k, v, q_scale, k_scale, v_scale, *, causal, softmax_scale=0.0, q_pos0=0, window=0,
                 softcap=0.0, q_fmt=E4M3, kv_fmt=E4M3, v_scale_axis=V_SCALES_ALONG_D, want_lse=False, device="cuda"):
        for t in (q, k, v, q_scale, k_scale, v_scale):
            if t.is_cuda or not t.is_contiguous():
                raise ValueError("host runner takes contiguous CPU tensors (pinned for full copy speed)")
        _check_prefill_tensors(q, k, v, q_scale, k_scale, v_scale, None, None, v_scale_axis)
        self.keep = (q, k, v, q_scale, k_scale, v_scale)
        B, H, S_q, d = q.shape
        self.o = torch.empty((B, H, S_q, d), dtype=torch.bfloat16).pin_memory()
        self.lse = torch.empty((B, H, S_q), dtype=torch.float32).pin_memory() if want_lse else None
        self.args = _prefill_args(q, k, v, q_scale, k_scale, v_scale, self.o, self.lse, causal, softmax_scale, q_pos0,
                                  window, softcap, q_fmt, kv_fmt, v_scale_axis)
        need = lib().rk_attn_prefill_host_arena_bytes(C.byref(self.args))
        self.arena = torch.empty(need + 1024, dtype=torch.uint8, device=device)
        self.h2d_bytes = sum(t.numel() * t.element_size() for t in self.keep)
        self.d2h_bytes = self.o.numel() * 2

    def run(self):
        check(lib().rk_attn_prefill_host(C.byref(self.args), _ptr(self.arena), self.arena.numel(), _stream()),
              "rk_attn_prefill_host")
        return self.o


def attn_prefill_host(q, k, v, q_scale, k_scale, v_scale, **kw):
    return PrefillHostRunner(q, k, v, q_scale, k_scale, v_scale, **kw).run()


def kv_cache_append(k_new, v_new, pos, k_codes, k_scales, v_codes, v_scales, fmt=E4M3):
    """Quantize one new K row and V row per (batch, KV head) (fp32 [B,H_kv,d]) into row pos[b] of the cache
    (codes [B,H_kv,L,d], scales [B,H_kv,L,d/32]); pos is an int32 CUDA tensor [B]."""
    front().kv_cache_append(k_new, v_new, pos, k_codes, k_scales, v_codes, v_scales, fmt)


def attn_decode_num_splits(B, H, H_kv, L, d=128, num_splits=0, kv_fmt=E4M3):
    a = DecodeArgs()
    a.B, a.H, a.H_kv, a.L, a.d, a.num_splits, a.kv_fmt = B, H, H_kv, L, d, num_splits, kv_fmt
    return lib().rk_attn_decode_num_splits(C.byref(a))


def attn_decode_workspace_bytes(B, H, H_kv, L, d=128, num_splits=0, kv_fmt=None):
    """Bytes of attn_decode's workspace for a cache format; without one, enough for each of them."""
    a = DecodeArgs()
    a.B, a.H, a.H_kv, a.L, a.d, a.num_splits = B, H, H_kv, L, d, num_splits
    sizes = []
    for a.kv_fmt in (E4M3, E2M1) if kv_fmt is None else (kv_fmt,):       # one format of each kernel
        sizes.append(lib().rk_attn_decode_workspace_bytes(C.byref(a)))
    return max(sizes)


def _check_decode_tensors(q, k, v, k_scale, v_scale, kv_len, out, lse):
    front().check_decode_tensors(q, k, v, k_scale, v_scale, kv_len, out, lse)


def attn_decode(q, k, v, k_scale, v_scale, *, kv_len=None, softmax_scale=0.0, kv_fmt=E4M3, num_splits=0, out=None,
                lse=None, workspace=None):
    """Decode attention: q bf16 [B,H,d]; k/v codes [B,H_kv,L,d]; scales [B,H_kv,L,d/32]; kv_len int32 [B] or None.
    Returns O bf16 [B,H,d]."""
    return front().attn_decode(q, k, v, k_scale, v_scale, kv_len, out, lse, workspace, softmax_scale, kv_fmt, num_splits)


def last_device_status():
    return lib().rk_last_device_status()


def shard_range(n_units, rank, world):
    """Contiguous block partition of n_units independent (batch, KV-head) units over `world` ranks (rk_shard_units)."""
    lo, hi = C.c_int64(), C.c_int64()
    check(lib().rk_shard_units(n_units, rank, world, C.byref(lo), C.byref(hi)), "rk_shard_units")
    return lo.value, hi.value
