"""Performance cases of the MX attention path: what a model's layer asks of this framework, through its Python entry
points, from the smallest call to the largest.

Four kinds of work:
  prefill  attn_prefill over quantized Q, K, V: whole prompts (S_kv = S_q) and chunks of a prompt behind a cached prefix
           (S_kv > S_q, the chunk's first row at global position S_kv - S_q)
  decode   one generation step of a batch: kv_cache_append of the step's new token, then attn_decode over the cache
  qkv      what a layer does between its QKV projection and attention: RoPE + quantization of Q and K, quantization of V
  norm     RMSNorm + quantization of the residual stream in front of a projection

Operands are N(0,1) fp32 (Gemma-style prefill: times 0.5) drawn from the seed and quantized by this library, the data
the repository's benchmark uses.
"""
import math

import torch

import radiance_kernels_b200 as rk

E4M3, E5M2, E2M3, E3M2, E2M1 = rk.E4M3, rk.E5M2, rk.E2M3, rk.E3M2, rk.E2M1


def _prefill(B, H, H_kv, S_q, S_kv, d, causal=True, window=0, softcap=0.0, mul=1.0, q_fmt=E4M3, kv_fmt=E4M3, v_along_keys=False):
    return dict(kind="prefill", B=B, H=H, H_kv=H_kv, S_q=S_q, S_kv=S_kv, d=d, causal=causal, window=window, softcap=softcap,
                mul=mul, q_fmt=q_fmt, kv_fmt=kv_fmt, v_along_keys=v_along_keys)


def _decode(B, H, H_kv, L, shortest, kv_fmt=E4M3):
    return dict(kind="decode", B=B, H=H, H_kv=H_kv, L=L, shortest=shortest, d=128, kv_fmt=kv_fmt)


def _qkv(B, H, H_kv, S, d, pos0=0, v_along_keys=False, v_bf16=False):
    return dict(kind="qkv", B=B, H=H, H_kv=H_kv, S=S, d=d, pos0=pos0, v_along_keys=v_along_keys, v_bf16=v_bf16)


def _norm(rows, K, bf16=True):
    return dict(kind="norm", rows=rows, K=K, bf16=bf16)


def listed():
    return [
        # The smallest call: one head over one short non-causal block (an encoder or a unit of a sharded job), bound by
        # launches and latency.
        dict(name="prefill_one_head_S256_d64", **_prefill(1, 1, 1, 256, 256, 64, causal=False)),
        # Chunked prefill of one request in a serving loop: a ragged chunk of a prompt behind its cached prefix.
        dict(name="prefill_chunk_509_of_3581", **_prefill(1, 32, 8, 509, 3581, 128)),
        # The repository's headline benchmark: a batch of prompts, MHA.
        dict(name="prefill_mha_B8_S4096", **_prefill(8, 16, 16, 4096, 4096, 128)),
        # Long prompts, grouped-query attention: the benchmark's GQA configuration, the largest prefill here.
        dict(name="prefill_gqa_B4_S8192", **_prefill(4, 32, 8, 8192, 8192, 128)),
        # Gemma-style heads: d = 256, logits soft-capped at 50.
        dict(name="prefill_gemma_cap50_S8192", **_prefill(2, 16, 8, 8192, 8192, 256, softcap=50.0, mul=0.5)),
        # The same heads with 6-bit operands (E2M3 Q, E3M2 K and V), codes one per byte as the quantizer writes them.
        dict(name="prefill_gemma_mxfp6_S8192", **_prefill(2, 16, 8, 8192, 8192, 256, softcap=50.0, mul=0.5, q_fmt=E2M3, kv_fmt=E3M2)),
        # One interactive user: a decode step at batch 1, bound by latency and launches.
        dict(name="decode_B1_L6000", **_decode(1, 32, 8, 8192, 6000)),
        # Continuous batching: sequences of very different lengths share a step.
        dict(name="decode_ragged_B16_L8192", **_decode(16, 32, 8, 8192, 1000)),
        # Eight query heads per KV head (a 70B-class layer), long contexts.
        dict(name="decode_wide_B32_L32768", **_decode(32, 64, 8, 32768, 32768)),
        # The repository's decode benchmark: 64 sequences of 32k keys, the largest cache.
        dict(name="decode_B64_L32768", **_decode(64, 32, 8, 32768, 32768)),
        # Prompt processing: Q and K rotated and quantized, V quantized along d as the KV cache keeps it.
        dict(name="qkv_B2_S4096", **_qkv(2, 32, 8, 4096, 128)),
        # Residual stream of the same prompts in front of the QKV projection, bf16.
        dict(name="norm_8192x4096_bf16", **_norm(8192, 4096)),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    kind = rng.choices(("prefill", "decode", "qkv", "norm"), (0.4, 0.35, 0.15, 0.1))[0]
    H_kv, group = rng.choice((1, 2, 4, 8)), rng.choice((1, 2, 4, 8))
    if kind == "prefill":
        d = rng.choices((64, 128, 256), (0.25, 0.5, 0.25))[0]
        S_q = _logint(rng, 16, 8192)
        S_kv = S_q + (_logint(rng, 1, 8192) if rng.random() < 0.5 else 0)
        causal = rng.random() < 0.85
        softcap = 50.0 if d == 256 and rng.random() < 0.7 else 0.0
        window = _logint(rng, 128, 4096) if causal and rng.random() < 0.2 else 0
        q_fmt, kv_fmt = rng.choices(((E4M3, E4M3), (E5M2, E5M2), (E2M3, E3M2), (E2M1, E2M1)), (0.7, 0.08, 0.14, 0.08))[0]
        v_along_keys = rng.random() < 0.25
        H = H_kv * group
        B = _logint(rng, 1, 8)
        while True:
            c = _prefill(B, H, H_kv, S_q, S_kv, d, causal, window, softcap, 0.5 if d == 256 else 1.0, q_fmt, kv_fmt, v_along_keys)
            if work(c)["flops"] <= 2.0e12:
                return c
            B, S_q, S_kv = (B // 2, S_q, S_kv) if B > 1 else (B, S_q // 2, S_kv // 2)
    if kind == "decode":
        kv_fmt = rng.choices((E4M3, E5M2, E3M2, E2M1), (0.75, 0.1, 0.1, 0.05))[0]
        L = 4 * _logint(rng, 32, 16384)
        B = min(_logint(rng, 1, 128), max(1, (64 * 8 * 32768) // (H_kv * L)))
        return _decode(B, H_kv * group, H_kv, L, _logint(rng, 1, L) if rng.random() < 0.6 else L, kv_fmt)
    if kind == "qkv":
        tokens = _logint(rng, 1, 16384)
        B = min(tokens, rng.choice((1, 1, 2, 4, 8)))
        v_along_keys = rng.random() < 0.3
        return _qkv(B, H_kv * group, H_kv, max(1, tokens // B), rng.choice((64, 128, 128, 256)), _logint(rng, 1, 4096) - 1, v_along_keys,
                    not v_along_keys and rng.random() < 0.5)
    rows = _logint(rng, 1, 16384)
    return _norm(rows, 32 * _logint(rng, 16, 384 if rows < 4096 else 128), rng.random() < 0.7)


def _visible_keys(c):
    """Sum over the query rows of the keys each may see."""
    if not c["causal"]:
        return c["S_q"] * c["S_kv"]
    p0, w = c["S_kv"] - c["S_q"], c["window"]
    return sum(min(p + 1, w) if w else p + 1 for p in range(p0, p0 + c["S_q"]))


def _lengths(c):
    """Cached keys per sequence, this step's token among them: spread evenly from the shortest to the cache's extent."""
    B, lo, hi = c["B"], c["shortest"], c["L"]
    return [lo + (hi - lo) * b // max(1, B - 1) for b in range(B)]


def _randn(gen, shape, mul=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * mul


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": c}
    if c["kind"] == "prefill":
        q = _randn(gen, (c["B"], c["H"], c["S_q"], c["d"]), c["mul"])
        k, v = (_randn(gen, (c["B"], c["H_kv"], c["S_kv"], c["d"]), c["mul"]) for _ in range(2))
        s["q"], s["q_scale"] = rk.mx_quantize(q, c["q_fmt"])
        s["k"], s["k_scale"] = rk.mx_quantize(k, c["kv_fmt"])
        s["v"], s["v_scale"] = (rk.mx_quantize_keys if c["v_along_keys"] else rk.mx_quantize)(v, c["kv_fmt"])
        s["opts"] = dict(causal=c["causal"], q_pos0=c["S_kv"] - c["S_q"], window=c["window"], softcap=c["softcap"], q_fmt=c["q_fmt"],
                         kv_fmt=c["kv_fmt"], v_scale_axis=rk.V_SCALES_ALONG_KEYS if c["v_along_keys"] else rk.V_SCALES_ALONG_D)
    elif c["kind"] == "decode":
        B, H_kv, L, d = c["B"], c["H_kv"], c["L"], c["d"]
        cache = []
        for _ in range(2):                         # K, then V; one sequence at a time keeps the fp32 copy small
            codes = torch.empty((B, H_kv, L, d), dtype=torch.uint8, device="cuda")
            scales = torch.empty((B, H_kv, L, d // 32), dtype=torch.uint8, device="cuda")
            for b in range(B):
                codes[b], scales[b] = rk.mx_quantize(_randn(gen, (H_kv, L, d)), c["kv_fmt"])
            cache += [codes, scales]
        s["k"], s["k_scale"], s["v"], s["v_scale"] = cache
        lens = torch.tensor(_lengths(c), dtype=torch.int32, device="cuda")
        s["kv_len"] = lens[torch.randperm(B, generator=gen, device="cuda")].contiguous()
        s["pos"] = s["kv_len"] - 1
        s["q"] = _randn(gen, (B, c["H"], d)).to(torch.bfloat16)
        s["k_new"], s["v_new"] = _randn(gen, (B, H_kv, d)), _randn(gen, (B, H_kv, d))
    elif c["kind"] == "qkv":
        B, S, d = c["B"], c["S"], c["d"]
        s["q"] = _randn(gen, (B, c["H"], S, d))
        s["k"], s["v"] = (_randn(gen, (B, c["H_kv"], S, d)) for _ in range(2))
        if c["v_bf16"]:
            s["v"] = s["v"].to(torch.bfloat16)
        inv = 10000.0 ** (-torch.arange(0, d, 2, dtype=torch.float64, device="cuda") / d)
        angle = torch.arange(c["pos0"] + S, dtype=torch.float64, device="cuda")[:, None] * inv[None, :]
        s["cos"], s["sin"] = angle.cos().float().contiguous(), angle.sin().float().contiguous()
    else:
        x = _randn(gen, (c["rows"], c["K"]))
        s["x"] = x.to(torch.bfloat16) if c["bf16"] else x
        s["gamma"] = 1.0 + 0.1 * _randn(gen, (c["K"],))
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "prefill":
        return rk.attn_prefill(s["q"], s["k"], s["v"], s["q_scale"], s["k_scale"], s["v_scale"], **s["opts"])
    if c["kind"] == "decode":
        rk.kv_cache_append(s["k_new"], s["v_new"], s["pos"], s["k"], s["k_scale"], s["v"], s["v_scale"], c["kv_fmt"])
        o = rk.attn_decode(s["q"], s["k"], s["v"], s["k_scale"], s["v_scale"], kv_len=s["kv_len"], kv_fmt=c["kv_fmt"])
        return o, s["k"], s["k_scale"], s["v"], s["v_scale"]
    if c["kind"] == "qkv":
        q, q_scale = rk.rope_mx_quantize(s["q"], s["cos"], s["sin"], pos0=c["pos0"])
        k, k_scale = rk.rope_mx_quantize(s["k"], s["cos"], s["sin"], pos0=c["pos0"])
        v, v_scale = rk.mx_quantize_keys(s["v"]) if c["v_along_keys"] else rk.mx_quantize(s["v"])
        return q, q_scale, k, k_scale, v, v_scale
    return rk.rmsnorm_mx_quantize(s["x"], s["gamma"], 1e-5)


def work(case):
    """Bytes each input and output needs once, operations of the visible (query, key) pairs."""
    c = case
    if c["kind"] == "prefill":
        q, kv = c["B"] * c["H"] * c["S_q"] * c["d"], c["B"] * c["H_kv"] * c["S_kv"] * c["d"]
        return {"bytes": (q + 2 * kv) * 33 / 32 + 2 * q, "flops": 4.0 * c["B"] * c["H"] * c["d"] * _visible_keys(c)}
    if c["kind"] == "decode":
        keys, qo = sum(_lengths(c)), c["B"] * c["H"] * c["d"]
        new = 2 * c["B"] * c["H_kv"] * c["d"]
        return {"bytes": 2 * keys * c["H_kv"] * c["d"] * 33 / 32 + 4 * qo + new * (4 + 33 / 32), "flops": 4.0 * keys * c["H"] * c["d"]}
    if c["kind"] == "qkv":
        qk, v = c["B"] * (c["H"] + c["H_kv"]) * c["S"] * c["d"], c["B"] * c["H_kv"] * c["S"] * c["d"]
        return {"bytes": qk * (4 + 33 / 32) + v * ((2 if c["v_bf16"] else 4) + 33 / 32) + 4 * c["S"] * c["d"], "flops": 5.0 * qk + 2.0 * v}
    n = c["rows"] * c["K"]
    return {"bytes": n * ((2 if c["bf16"] else 4) + 33 / 32) + 4 * c["K"], "flops": 5.0 * n}


def tolerance(case):
    """Codes and scales are the same bit for bit.  Attention returns bf16 from 8-bit (or narrower) operands with fp32
    accumulation; another order of the sums moves O by well under a bf16 step, and now and then one requantized P by one of
    its steps."""
    return "exact" if case["kind"] in ("qkv", "norm") else {"rel": 1e-2}
