"""Decode attention over an MXFP8 KV cache against the CPU oracle, through the C ABI."""
import numpy as np
import pytest
import torch

import oracle
import radiance_kernels_b200 as rk
from helpers import MAX_ABS, REL_L2, errors, np_

pytestmark = pytest.mark.gpu


def run(B, H, Hkv, L, lens=None, seed=0, num_splits=0, want_lse=False, vmul=1.0, kv_fmt=rk.E4M3):
    d = 128
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(B, H, d, generator=g, device="cuda").bfloat16()
    K = torch.randn(B, Hkv, L, d, generator=g, device="cuda")
    V = torch.randn(B, Hkv, L, d, generator=g, device="cuda") * vmul
    kc, ks = rk.mx_quantize(K, kv_fmt)
    vc, vs = rk.mx_quantize(V, kv_fmt)
    kl = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    lse = torch.empty(B, H, dtype=torch.float32, device="cuda") if want_lse else None
    o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=kl, num_splits=num_splits, lse=lse, kv_fmt=kv_fmt)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    ref = oracle.attn_decode(np_(q.view(torch.uint16)), np_(kc), np_(vc), np_(ks), np_(vs), softmax_scale=d ** -0.5,
                             kv_len=None if lens is None else np.array(lens, np.int32), want_lse=want_lse, kv_fmt=kv_fmt)
    got = np_(o.float())
    assert np.isfinite(got).all()
    ma, rl = errors(got, ref["o_f32"])
    big = max(1.0, float(np.abs(ref["o_f32"]).max()))        # output magnitudes follow V's: the absolute bound with them
    assert ma <= MAX_ABS * big and rl <= REL_L2, (ma, rl)
    if want_lse:
        assert np.abs(np_(lse) - ref["lse"]).max() < 2e-3
    return got, ref


@pytest.mark.parametrize("grp", [1, 2, 4, 8])
def test_group_sizes(grp):
    run(2, 2 * grp, 2, 1024, seed=grp)


@pytest.mark.parametrize("grp", [1, 4, 8])
def test_e5m2_cache(grp):
    """An E5M2 cache (what rk_kv_cache_append writes with fmt = RK_FMT_E5M2): the tcgen05 kernel feeds the raw tiles
    to block-scaled MMAs, so the cache format is one field of the instruction descriptor."""
    run(2, 2 * grp, 2, 2048, seed=60 + grp, kv_fmt=rk.E5M2, want_lse=True)
    run(2, 2 * grp, 2, 1000, lens=[1000, 37], seed=70 + grp, kv_fmt=rk.E5M2)


@pytest.mark.parametrize("fmt", [rk.E2M3, rk.E3M2, rk.E2M1])
def test_six_and_four_bit_caches(fmt):
    """Caches in the 6-bit and 4-bit formats rk_kv_cache_append can write (one code per byte): the tensor core does
    not read that form, so these go through the kernel whose threads convert the codes (hardware conversions to f16 for
    K, bit placement into bf16 for V)."""
    run(2, 8, 2, 2048, seed=80 + fmt, kv_fmt=fmt, want_lse=True)
    run(2, 16, 2, 1000, lens=[1000, 37], seed=90 + fmt, kv_fmt=fmt)
    run(1, 2, 2, 512, seed=95 + fmt, kv_fmt=fmt, vmul=300.0)            # large V block scales


def test_e5m2_cache_through_the_converting_kernel():
    """The same E5M2 cache through the mma.sync kernel (test hook), which is templated on the cache format."""
    try:
        rk.lib().rk_debug_set_decode_path(1)
        run(2, 8, 2, 2048, seed=61, kv_fmt=rk.E5M2, want_lse=True)
    finally:
        rk.lib().rk_debug_set_decode_path(0)


def test_llama_shape_small_batch():
    """32 query heads on 8 KV heads, d=128 (the benchmark's head geometry) at a length the oracle finishes fast."""
    run(2, 32, 8, 4096, seed=1)


def test_ragged_kv_len_and_splits():
    run(3, 8, 2, 4096, lens=[4096, 1, 2500], seed=2)
    run(2, 8, 2, 1000, lens=[1000, 37], seed=3)
    run(1, 4, 1, 2048, num_splits=1, seed=4)
    run(1, 4, 1, 2048, num_splits=16, seed=4)       # more splits than needed: some are short or empty
    run(1, 4, 1, 132, lens=[129], num_splits=2, seed=5)


def test_empty_and_tiny_sequences():
    """kv_len 0 gives O = 0 and LSE = -inf (the l <= 0 guard); lengths below one key tile and one key short of it."""
    g = torch.Generator(device="cuda").manual_seed(12)
    q = torch.randn(4, 8, 128, generator=g, device="cuda").bfloat16()
    K = torch.randn(4, 2, 256, 128, generator=g, device="cuda")
    V = torch.randn(4, 2, 256, 128, generator=g, device="cuda")
    kc, ks = rk.mx_quantize(K); vc, vs = rk.mx_quantize(V)
    lens = [0, 5, 127, 129]
    kl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    lse = torch.empty(4, 8, dtype=torch.float32, device="cuda")
    o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=kl, lse=lse)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    ref = oracle.attn_decode(np_(q.view(torch.uint16)), np_(kc), np_(vc), np_(ks), np_(vs), softmax_scale=128 ** -0.5,
                             kv_len=np.array(lens, np.int32), want_lse=True)
    got = np_(o.float())
    assert np.all(got[0] == 0.0) and np.all(np.isneginf(np_(lse)[0]))
    ma, rl = errors(got, ref["o_f32"])
    assert ma <= MAX_ABS and rl <= REL_L2, (ma, rl)
    assert np.abs(np_(lse)[1:] - ref["lse"][1:]).max() < 2e-3


def test_split_count_does_not_change_result_much():
    a, _ = run(1, 8, 2, 8192, num_splits=1, seed=6)
    b, _ = run(1, 8, 2, 8192, num_splits=8, seed=6)
    assert np.abs(a - b).max() < 4e-3


def test_lse_output():
    run(1, 8, 2, 1024, want_lse=True, seed=7)


@pytest.mark.parametrize("top_code", [134, 135, 200, 60])
def test_v_scale_codes_at_and_beyond_the_bf16_folding_edge(top_code):
    """V block scales whose largest code is 134 (the last one a fixed 2^120 folding constant can take in bf16), 135,
    200 and a very small 60, mixed with codes up to 24 below it inside every block of 32 keys: both decode kernels
    must re-centre the factor they fold into P and match the oracle.  Output magnitudes follow the scale, so the
    absolute bound is relative to the reference's largest value."""
    g = torch.Generator(device="cuda").manual_seed(40 + top_code)
    q = torch.randn(2, 8, 128, generator=g, device="cuda").bfloat16()
    kc, ks, vc, vs = _quantized_cache(2, 2, 1024, seed=41 + top_code)
    vs = torch.randint(top_code - 24, top_code + 1, vs.shape, generator=g, dtype=torch.uint8, device="cuda")
    vs[:, :, 5::97] = top_code                      # the top code is present in every sequence
    (legacy, tc), ref = _check(q, kc, ks, vc, vs)
    big = float(np.abs(ref["o_f32"]).max())
    assert np.abs(legacy - tc).max() <= 1e-2 * max(1.0, big)      # one bf16 step of the output at that magnitude


def test_full_length_one_sequence():
    """KV length 32768 (the benchmark's per-sequence length) for one sequence, all 8 KV heads."""
    run(1, 32, 8, 32768, seed=9)


def _quantized_cache(B, Hkv, L, seed, kmul=1.0, vscale_spread=0):
    d = 128
    g = torch.Generator(device="cuda").manual_seed(seed)
    K = torch.randn(B, Hkv, L, d, generator=g, device="cuda") * kmul
    V = torch.randn(B, Hkv, L, d, generator=g, device="cuda")
    if vscale_spread:       # per-key magnitudes spread over 2^+-spread: block scales differ widely inside a 32-key block
        e = torch.randint(-vscale_spread, vscale_spread + 1, (B, Hkv, L, 1), generator=g, device="cuda").float()
        V = V * torch.exp2(e)
    kc, ks = rk.mx_quantize(K)
    vc, vs = rk.mx_quantize(V)
    return kc, ks, vc, vs


def _check(q, kc, ks, vc, vs, lens=None, num_splits=0):
    d = 128
    kl = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    ref = oracle.attn_decode(np_(q.view(torch.uint16)), np_(kc), np_(vc), np_(ks), np_(vs), softmax_scale=d ** -0.5,
                             kv_len=None if lens is None else np.array(lens, np.int32))
    outs = []
    for path in (1, 0):                       # 1 = the mma.sync kernel, 0 = chosen by shape (tcgen05 for these shapes)
        rk.lib().rk_debug_set_decode_path(path)
        try:
            o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=kl, num_splits=num_splits)
            torch.cuda.synchronize()
        finally:
            rk.lib().rk_debug_set_decode_path(0)
        assert rk.last_device_status() == 0
        got = np_(o.float())
        assert np.isfinite(got).all(), f"path {path}: non-finite output"
        ma, rl = errors(got, ref["o_f32"])
        # the absolute bound is stated for outputs of order one; scale it with the reference's magnitude
        assert ma <= MAX_ABS * max(1.0, float(np.abs(ref["o_f32"]).max())) and rl <= REL_L2, (path, ma, rl)
        outs.append(got)
    return outs, ref


def test_both_decode_kernels_match_the_oracle():
    g = torch.Generator(device="cuda").manual_seed(21)
    q = torch.randn(2, 8, 128, generator=g, device="cuda").bfloat16()
    kc, ks, vc, vs = _quantized_cache(2, 2, 2048, seed=22)
    (legacy, tc), ref = _check(q, kc, ks, vc, vs)
    assert np.abs(legacy - tc).max() < 4e-3


def test_tc_decode_peaked_rows_and_growing_maxima():
    """Large logits: a few keys dominate, the running maximum keeps growing along the sequence (keys scaled up
    towards the end), so O is rescaled several times and most p are far below the block maximum."""
    g = torch.Generator(device="cuda").manual_seed(23)
    q = (torch.randn(1, 4, 128, generator=g, device="cuda") * 4.0).bfloat16()
    kc, ks, vc, vs = _quantized_cache(1, 1, 4096, seed=24)
    K = torch.randn(1, 1, 4096, 128, generator=g, device="cuda") * torch.linspace(0.2, 3.0, 4096, device="cuda").view(1, 1, -1, 1)
    kc, ks = rk.mx_quantize(K)
    _check(q, kc, ks, vc, vs, num_splits=1)
    _check(q, kc, ks, vc, vs, num_splits=4)


def test_tc_decode_v_scales_spread_inside_a_block():
    g = torch.Generator(device="cuda").manual_seed(25)
    q = torch.randn(1, 8, 128, generator=g, device="cuda").bfloat16()
    kc, ks, vc, vs = _quantized_cache(1, 2, 1024, seed=26, vscale_spread=12)
    _check(q, kc, ks, vc, vs)


def test_decode_ignores_poisoned_cache_past_kv_len():
    """Keys at and beyond kv_len hold NaN codes and NaN scales (0x7F / 0xFF): they must not reach the result."""
    g = torch.Generator(device="cuda").manual_seed(27)
    q = torch.randn(2, 8, 128, generator=g, device="cuda").bfloat16()
    kc, ks, vc, vs = _quantized_cache(2, 2, 1024, seed=28)
    lens = [700, 130]
    clean = [t.clone() for t in (kc, ks, vc, vs)]
    for b, n in enumerate(lens):
        kc[b, :, n:] = 0x7F; vc[b, :, n:] = 0x7F; ks[b, :, n:] = 0xFF; vs[b, :, n:] = 0xFF
    kl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    ref = oracle.attn_decode(np_(q.view(torch.uint16)), np_(clean[0]), np_(clean[2]), np_(clean[1]), np_(clean[3]),
                             softmax_scale=128 ** -0.5, kv_len=np.array(lens, np.int32))
    o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=kl)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    got = np_(o.float())
    assert np.isfinite(got).all()
    ma, rl = errors(got, ref["o_f32"])
    assert ma <= MAX_ABS and rl <= REL_L2, (ma, rl)


@pytest.mark.parametrize("fmt", [rk.E4M3, rk.E3M2, rk.E2M1])
def test_kv_cache_append_then_decode_in_a_loop(fmt):
    """Tokens appended one at a time give the cache that quantizing the whole tensor gives (bit for bit, and equal
    to the CPU oracle's rows); decode over the growing cache matches the oracle at every length tried.  Every format
    the append kernel writes is one the decode entry point reads."""
    B, Hkv, H, L, d, T = 2, 2, 8, 160, 128, 150
    g = torch.Generator(device="cuda").manual_seed(31)
    K = torch.randn(B, Hkv, L, d, generator=g, device="cuda")
    V = torch.randn(B, Hkv, L, d, generator=g, device="cuda") * 3.0
    q = torch.randn(B, H, d, generator=g, device="cuda").bfloat16()
    kc_all, ks_all = rk.mx_quantize(K, fmt)
    vc_all, vs_all = rk.mx_quantize(V, fmt)
    kc = torch.full((B, Hkv, L, d), 0x7F, dtype=torch.uint8, device="cuda")      # unwritten rows are poison
    vc = torch.full_like(kc, 0x7F)
    ks = torch.full((B, Hkv, L, d // 32), 0xFF, dtype=torch.uint8, device="cuda")
    vs = torch.full_like(ks, 0xFF)
    lens = [0, 0]
    for t in range(T):
        pos = torch.tensor([t, t if t < 100 else -1], dtype=torch.int32, device="cuda")   # sequence 1 stops at 100 tokens
        rk.kv_cache_append(K[:, :, t].contiguous(), V[:, :, t].contiguous(), pos, kc, ks, vc, vs, fmt=fmt)
        lens = [t + 1, min(t + 1, 100)]
        if t in (0, 31, 99, 127, 128, T - 1):
            kl = torch.tensor(lens, dtype=torch.int32, device="cuda")
            o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=kl, kv_fmt=fmt)
            torch.cuda.synchronize()
            assert rk.last_device_status() == 0
            ref = oracle.attn_decode(np_(q.view(torch.uint16)), np_(kc_all), np_(vc_all), np_(ks_all), np_(vs_all),
                                     softmax_scale=d ** -0.5, kv_len=np.array(lens, np.int32), kv_fmt=fmt)
            got = np_(o.float())
            assert np.isfinite(got).all()
            ma, rl = errors(got, ref["o_f32"])
            assert ma <= MAX_ABS * 3.0 and rl <= REL_L2, (t, ma, rl)
    assert torch.equal(kc[0, :, :T], kc_all[0, :, :T]) and torch.equal(ks[0, :, :T], ks_all[0, :, :T])
    assert torch.equal(vc[0, :, :T], vc_all[0, :, :T]) and torch.equal(vs[0, :, :T], vs_all[0, :, :T])
    assert torch.equal(kc[1, :, :100], kc_all[1, :, :100]) and bool((kc[1, :, 100:] == 0x7F).all())
    oc, os_ = oracle.quantize(np_(V[0, 0, :T]), axis=1, fmt=fmt)
    assert np.array_equal(np_(vc[0, 0, :T]), oc) and np.array_equal(np_(vs[0, 0, :T]), os_)


# 0 sequences: as many as it takes for a second pass of the append kernel's grid (four CTAs of 128 threads per SM for K and as many for V, 8 elements a thread)
@pytest.mark.parametrize("B,Hkv,L,d,fmt", [(1, 1, 1, 32, rk.E4M3), (3, 5, 2, 96, rk.E5M2), (7, 3, 4, 64, rk.E2M1), (33, 1, 3, 160, rk.E2M3), (5, 2, 300, 256, rk.E3M2),
                                           (0, 2, 3, 128, rk.E4M3), (0, 3, 2, 96, rk.E3M2), (0, 1, 2, 32, rk.E4M3)])
def test_kv_cache_append_writes_the_rows_it_is_given_and_no_other(B, Hkv, L, d, fmt):
    """Row widths that are no power of two, numbers of chunks that do not fill a warp, one thread's second row; positions outside the cache are skipped; rows of
    zeros and blocks with a NaN or an infinity among the new ones."""
    if B == 0:
        B = -(-(torch.cuda.get_device_properties(0).multi_processor_count * 4 * 128 + 77) * 8 // (Hkv * d))
    rng = np.random.default_rng(B + d)
    new = [(rng.standard_normal((B, Hkv, d)) * np.exp2(rng.integers(-8, 9, (B, Hkv, 1)))).astype(np.float32) for _ in range(2)]
    new[0][B // 2, 0] = 0.0
    if B > 2:
        new[0][B - 1, Hkv - 1, d - 1] = np.inf
        new[1][0, 0, 3] = np.nan
    pos = rng.integers(0, L, B).astype(np.int32)
    pos[1::7], pos[2::7], pos[4::7] = -1, L, 2 ** 31 - 1
    cache = [torch.full((B, Hkv, L, n), 0xA5, dtype=torch.uint8, device="cuda") for n in (d, d // 32) * 2]
    rk.kv_cache_append(*(torch.from_numpy(x).cuda() for x in new), torch.from_numpy(pos).cuda(), *cache, fmt=fmt)
    torch.cuda.synchronize()
    inside = np.flatnonzero((pos >= 0) & (pos < L))
    for x, got in zip(new, (cache[:2], cache[2:])):
        for part, rows in zip(got, oracle.quantize(x.reshape(B * Hkv, d), fmt)):
            want = np.full(part.shape, 0xA5, np.uint8)
            want[inside, :, pos[inside]] = rows.reshape(B, Hkv, -1)[inside]
            assert np.array_equal(np_(part), want)


@pytest.mark.parametrize("grp,case", [(4, "short"), (8, "short"), (4, "many"), (8, "many"), (4, "rising"), (8, "rising"), (4, "v jump"), (8, "v jump"), (1, "few tiles")])
def test_ranges_and_references(grp, case):
    """The tcgen05 kernel's equal ranges of tiles and its running references: a few and many short sequences per CTA (empty ones,
    single keys and tile edges among them), fewer tiles than CTAs, scores that rise by far more than 2^32 over the keys and V block
    scales that do (O is then rescaled, again and again, while other tiles are in flight)."""
    Hkv, d = 2, 128
    B, L = {"short": (71, 520), "many": (900, 260), "rising": (2, 3000), "v jump": (2, 3000), "few tiles": (3, 132)}[case]
    rng = np.random.default_rng(grp)
    lens = rng.choice([n for n in (0, 1, 127, 128, 129, 256, 384, 520) if n <= L], B).astype(np.int32) if B > 3 else np.array([L, 0, 5] if B == 3 else [L, L - 77], np.int32)
    g = torch.Generator(device="cuda").manual_seed(grp)
    q = torch.randn(B, grp * Hkv, d, generator=g, device="cuda").bfloat16()
    K = torch.randn(B, Hkv, L, d, generator=g, device="cuda")
    V = torch.randn(B, Hkv, L, d, generator=g, device="cuda")
    step = torch.arange(L, device="cuda", dtype=torch.float32).view(1, 1, L, 1) / L
    if case == "rising":
        K = K * 0.25 + step * 40.0 * q.float().view(B, Hkv, grp, d)[:, :, :1].sign()      # the first head of a group climbs by some 500
    if case == "v jump":
        V = V * torch.exp2(torch.floor(step * 100.0 - 60.0))
    kc, ks = rk.mx_quantize(K)
    vc, vs = rk.mx_quantize(V)
    lse = torch.empty(B, grp * Hkv, dtype=torch.float32, device="cuda")
    o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=torch.from_numpy(lens).cuda(), lse=lse)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    ref = oracle.attn_decode(np_(q.view(torch.uint16)), np_(kc), np_(vc), np_(ks), np_(vs), softmax_scale=d ** -0.5, kv_len=lens, want_lse=True)
    got, want = np_(o.float()), ref["o_f32"]
    assert np.isfinite(got).all()
    big = max(1.0, float(np.abs(want).max()))
    assert np.abs(got - want).max() <= MAX_ABS * big and errors(got, want)[1] <= REL_L2
    full = lens > 0
    assert np.abs(np_(lse)[full] - ref["lse"][full]).max() < 2e-3
    assert (got[~full] == 0).all()


@pytest.mark.parametrize("grp,kmul,lens", [(4, 1.0, [1, 1, 1, 1]), (8, 300.0, [3000, 1000, 129, 2]), (4, 3.0e7, [3000, 1000, 129, 1]), (1, 1.0e9, [3000, 700, 300, 5])])
def test_a_key_with_all_the_weight_gives_its_v_row_exactly(grp, kmul, lens):
    """One key is all a row sees, or its score lies 30 above every other one (scores up to 1e10): the p of the largest score is 1,
    which the two MXFP8 terms of P hold exactly, so O is the key's decoded V, bit for bit (an E4M3 code times a power of two is
    a bf16; the other keys add less than e^-30)."""
    B, Hkv, L, d = len(lens), 2, max(lens) // 4 * 4 + 4, 128
    g = torch.Generator(device="cuda").manual_seed(grp)
    q = torch.randn(B, grp * Hkv, d, generator=g, device="cuda").bfloat16()
    kc, ks, vc, vs = _quantized_cache(B, Hkv, L, seed=50 + grp, kmul=kmul)
    o = rk.attn_decode(q, kc, vc, ks, vs, kv_len=torch.tensor(lens, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    k, v = _decoded(kc, ks), _decoded(vc, vs)
    seen = 0
    for b in range(B):
        s = torch.einsum("hgd,hkd->hgk", q[b].double().view(Hkv, grp, d), k[b, :, :lens[b]]) * d ** -0.5
        top, at = s.topk(min(2, lens[b]), -1)
        for h in range(Hkv):
            for x in range(grp):
                if lens[b] == 1 or top[h, x, 0] - top[h, x, 1] > 30:
                    seen += 1
                    assert torch.equal(o[b, h * grp + x].double(), v[b, h, at[h, x, 0]]), (b, h, x)
    assert seen >= B * Hkv * grp // 2


def _decoded(codes, scales):
    return codes.view(torch.float8_e4m3fn).double() * torch.exp2(scales.double() - 127).repeat_interleave(32, -1)


def _error_beyond_rounding(o, q, kc, ks, vc, vs):
    """Relative 2-norm of O's error against 64 bits, and what of it exceeds that of rounding the exact O to bf16."""
    (B, H, d), Hkv = q.shape, kc.shape[1]
    want = torch.empty(B, H, d, dtype=torch.float64, device="cuda")
    for b in range(B):
        s = torch.einsum("hgd,hkd->hgk", q[b].double().view(Hkv, H // Hkv, d), _decoded(kc[b], ks[b])) * d ** -0.5
        want[b] = torch.einsum("hgk,hkd->hgd", torch.softmax(s, -1), _decoded(vc[b], vs[b])).reshape(H, d)
    rel = float((o.double() - want).norm() / want.norm())
    rounding = float((want.float().bfloat16().double() - want).norm() / want.norm())
    return rel, max(rel ** 2 - rounding ** 2, 0.0) ** 0.5


@pytest.mark.parametrize("grp", [4, 8])
def test_error_of_peaked_rows(grp):
    """Queries of twelve times unit variance: most of the weight lies on a key or two, and its error is that of their p.  Beyond
    the rounding of O to bf16 there are 4.1e-4 with the p of the largest score exact (5.8e-4 with one rounded like all others)."""
    g = torch.Generator(device="cuda").manual_seed(51)
    q = (torch.randn(32, 8 * grp, 128, generator=g, device="cuda") * 12.0).bfloat16()
    kc, ks, vc, vs = _quantized_cache(32, 8, 4096, seed=52)
    rel, beyond = _error_beyond_rounding(rk.attn_decode(q, kc, vc, ks, vs), q, kc, ks, vc, vs)
    assert rk.last_device_status() == 0
    assert beyond <= 5.0e-4, (rel, beyond)


@pytest.mark.parametrize("grp", [4, 8])
@pytest.mark.parametrize("octaves,bound", [(4, 7e-4), (5, 7e-4), (8, 7e-4), (12, 4.5e-3)])
def test_error_where_light_keys_have_the_large_v_scales(octaves, bound, grp):
    """One key in 32 has V scales some octaves above the others' and next to no weight: the weights of the others, moved down by
    those octaves, must keep their bits.  Two E4M3 terms reach down to 2^-22 of a block's largest element; the errors beyond
    rounding that this leaves are 6.1e-4, 6.1e-4, 6.2e-4 and 3.6e-3 (codes moved without rounding into the subnormals, 2^-15: 6.1e-4,
    8e-4, 1.4e-2, 0.31)."""
    g = torch.Generator(device="cuda").manual_seed(53)
    B, Hkv, L, d = 32, 8, 1024, 128
    q = torch.randn(B, Hkv * grp, d, generator=g, device="cuda").bfloat16()
    K, V = (torch.randn(B, Hkv, L, d, generator=g, device="cuda") for _ in range(2))
    first = q.view(B, Hkv, grp, d)[:, :, :1]                       # of every group of heads: the one the light keys are made for
    K[:, :, ::32] -= 3.0 * first.float()
    V[:, :, ::32] *= 2.0 ** octaves
    kc, ks = rk.mx_quantize(K)
    vc, vs = rk.mx_quantize(V)
    o = rk.attn_decode(q, kc, vc, ks, vs).view(B, Hkv, grp, d)[:, :, 0]
    assert rk.last_device_status() == 0
    rel, beyond = _error_beyond_rounding(o, first[:, :, 0], kc, ks, vc, vs)
    assert beyond <= bound, (rel, beyond)


@pytest.mark.parametrize("fmt,code", [(rk.E4M3, 0x7F), (rk.E4M3, 0xFF), (rk.E5M2, 0x7C), (rk.E5M2, 0x7F)])
@pytest.mark.parametrize("grp,num_splits", [(4, 0), (8, 0), (4, 3)])
def test_a_nan_score_reaches_every_column(grp, num_splits, fmt, code):
    """One key inside kv_len with a NaN (or, in E5M2, an infinity) among its codes and V scales below its neighbours': the score is
    no number, so no column of O is one, nor the log-sum-exp, wherever the unit's tiles were cut; other units are untouched."""
    B, Hkv, L, d = 3, 2, 3000, 128
    g = torch.Generator(device="cuda").manual_seed(57)
    q = torch.randn(B, Hkv * grp, d, generator=g, device="cuda").bfloat16()
    q[:, :, 17] = 1.0                                              # (a negative query element would make an infinity a score of -inf)
    K, V = (torch.randn(B, Hkv, L, d, generator=g, device="cuda") for _ in range(2))
    hit = [(0, 0, 5), (0, 1, 2999), (2, 0, 1290)]
    for octaves, (b, h, k) in zip((-2, -4, -11), hit):
        V[b, h, k] *= 2.0 ** octaves
        V[b, h, k, 32:64] *= 2.0 ** octaves
    kc, ks = rk.mx_quantize(K, fmt)
    vc, vs = rk.mx_quantize(V, fmt)
    kw = dict(kv_fmt=fmt, num_splits=num_splits)
    lse = torch.empty(2, B, Hkv * grp, dtype=torch.float32, device="cuda")
    clean = rk.attn_decode(q, kc, vc, ks, vs, lse=lse[0], **kw).view(B, Hkv, grp, d)
    for b, h, k in hit:
        kc[b, h, k, 17] = code
    o = rk.attn_decode(q, kc, vc, ks, vs, lse=lse[1], **kw).view(B, Hkv, grp, d)
    assert rk.last_device_status() == 0
    lse = lse.view(2, B, Hkv, grp)
    for b in range(B):
        for h in range(Hkv):
            if any((b, h) == at[:2] for at in hit):
                assert o[b, h].isnan().all() and lse[1, b, h].isnan().all(), (b, h)
            else:
                assert torch.equal(o[b, h], clean[b, h]) and torch.equal(lse[1, b, h], lse[0, b, h]), (b, h)


@pytest.mark.parametrize("fmt", [rk.E4M3, rk.E5M2, rk.E2M3, rk.E3M2, rk.E2M1])
@pytest.mark.parametrize("B,H,Hkv,L,num_splits", [(1, 8, 2, 8192, 0), (1, 4, 4, 2048, 0), (40, 8, 2, 640, 0), (2, 8, 2, 1000, 3)])
def test_workspaces_sized_by_the_helpers(B, H, Hkv, L, num_splits, fmt):
    """A workspace of the helper's size without a format, of its size for the format, and of one partial per split and head
    (fewer ranges then): each is taken, nothing is written past it, and the outputs agree."""
    g = torch.Generator(device="cuda").manual_seed(58)
    q = torch.randn(B, H, 128, generator=g, device="cuda").bfloat16()
    kc, ks = rk.mx_quantize(torch.randn(B, Hkv, L, 128, generator=g, device="cuda"), fmt)
    vc, vs = rk.mx_quantize(torch.randn(B, Hkv, L, 128, generator=g, device="cuda"), fmt)
    kw = dict(kv_fmt=fmt, num_splits=num_splits)
    want = rk.attn_decode(q, kc, vc, ks, vs, **kw).float()
    shape = dict(B=B, H=H, H_kv=Hkv, L=L, num_splits=num_splits)
    for size in (rk.attn_decode_workspace_bytes(**shape), rk.attn_decode_workspace_bytes(**shape, kv_fmt=fmt),
                 B * H * rk.attn_decode_num_splits(**shape, kv_fmt=fmt) * 130 * 4):
        buf = torch.full((size + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        got = rk.attn_decode(q, kc, vc, ks, vs, workspace=buf[:size], **kw).float()
        assert bool((buf[size:] == 0xA5).all())
        assert float((got - want).norm() / want.norm()) < 4e-3           # another cut: each side within a bf16 rounding of the exact O
    with pytest.raises(rk.RkError):
        rk.attn_decode(q, kc, vc, ks, vs, workspace=buf[:256], **kw)
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("B,H,Hkv,L,lens", [(1, 8, 2, 20000, [90]), (1, 8, 2, 20000, [128 * 74]), (1, 8, 2, 20000, [128 * 74 + 1]), (3, 16, 2, 20000, [0, 700, 129]),
                                            (1, 4, 1, 512, None), (1, 4, 4, 4864, None)])
def test_fewer_key_tiles_than_ctas(B, H, Hkv, L, lens):
    """As many ranges as there are key tiles, as many tiles as SMs (148) and two more; CTAs without a range beside them, with lengths and without."""
    run(B, H, Hkv, L, lens=lens, seed=17 + B + L, want_lse=lens is None)
