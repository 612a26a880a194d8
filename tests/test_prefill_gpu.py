"""Prefill attention on the GPU against the CPU oracle (same block_n, same P rule), through the C ABI."""
import numpy as np
import pytest
import torch

import oracle
import radiance_kernels_b200 as rk
from helpers import MAX_ABS, PAIRS, REL_L2, SPLIT, TURNS, chosen_form, errors, np_, prefill_form, prefill_vs_oracle, quantize_inputs, randn_qkv

pytestmark = pytest.mark.gpu


def _check(r):
    ma, rl = r["err"]
    assert ma <= MAX_ABS and rl <= REL_L2, (ma, rl)


def test_config1_single_head_noncausal_d64():
    """B=1 H=1 S=256 d=64 non-causal: the reference's own CPU-runnable case."""
    for seed in (0, 1, 2):
        _check(prefill_vs_oracle(1, 1, 1, 256, 256, 64, causal=False, seed=seed))


def test_single_tile_d128():
    _check(prefill_vs_oracle(1, 1, 1, 128, 128, 128, causal=False))


def test_causal_mha_d128():
    _check(prefill_vs_oracle(2, 4, 4, 1024, 1024, 128, causal=True, seed=1))


def test_causal_gqa_d128_group4():
    _check(prefill_vs_oracle(1, 8, 2, 768, 768, 128, causal=True, seed=2))


def test_reference_gqa_shape():
    """The reference's GQA kernel shape: 8 query heads on 2 KV heads, Sq=64 Sk=256 d=64, q_pos0=64
    (kernels/regen_data.sh:31-32)."""
    _check(prefill_vs_oracle(1, 8, 2, 64, 256, 64, causal=True, q_pos0=64, seed=0))


def test_gemma_softcap_d256():
    _check(prefill_vs_oracle(1, 4, 2, 512, 512, 256, causal=True, softcap=50.0, mul=0.5, seed=3))


def test_gemma_reference_style_cap_bites_window():
    """Q scaled by 50 so the cap saturates, sliding window 128, d=256, 8:4 heads
    (kernels/flash_attention_mx_gemma/fa_gen_data.py:77-79, kernels/regen_data.sh:33-34)."""
    _check(prefill_vs_oracle(1, 8, 4, 256, 512, 256, causal=True, softcap=50.0, qmul=50.0, q_pos0=256, window=128))


@pytest.mark.parametrize("d", [128, 256])
def test_softcap_scores_on_both_sides_of_the_series_limit(d):
    """The capped kernels evaluate tanh by its series while a warp's scores of a key tile stay below cap / 8 and by
    the exponential form otherwise: with Q scaled by 1.6 the largest |score| of a tile lies around that limit
    (6.25 at cap 50), so both forms run inside one launch and must meet the oracle's tanh."""
    _check(prefill_vs_oracle(1, 4, 2, 640, 640, d, causal=True, softcap=50.0, qmul=1.6, seed=23))
    _check(prefill_vs_oracle(1, 2, 2, 384, 384, d, causal=False, softcap=30.0, qmul=1.0, seed=24))


def test_sliding_window_d128():
    _check(prefill_vs_oracle(1, 2, 1, 640, 640, 128, causal=True, window=200, seed=4))


@pytest.mark.parametrize("d,S,window,q_pos0,softcap", [(128, 1536, 300, 0, 0.0), (128, 1100, 128, 700, 0.0),
                                                      (256, 1280, 200, 0, 50.0), (128, 900, 1, 0, 0.0)])
def test_sliding_window_skips_key_tiles_below_the_window(d, S, window, q_pos0, softcap):
    """Long sequences with a short window: most key tiles lie wholly below the window and are never loaded; the
    result must equal the oracle's, which masks them (d = 128 in every form; d = 256)."""
    for H in (2, 20) if d == 128 else (2,):
        _check(prefill_vs_oracle(1, H, 1, S, S + q_pos0, d, causal=True, window=window, q_pos0=q_pos0, softcap=softcap,
                                 mul=0.5 if d == 256 else 1.0, seed=60 + window))


def test_ragged_lengths_and_offset():
    _check(prefill_vs_oracle(1, 2, 2, 200, 333, 128, causal=True, q_pos0=133, seed=5))
    _check(prefill_vs_oracle(1, 1, 1, 1, 97, 64, causal=False, seed=6))
    _check(prefill_vs_oracle(1, 2, 1, 130, 31, 128, causal=False, seed=7))


def test_rows_without_visible_keys_are_zero():
    """q_pos0 < 0: the first rows see no key at all -> O = 0 (the l <= 0 guard of finalize_O)."""
    r = prefill_vs_oracle(1, 1, 1, 256, 256, 128, causal=True, q_pos0=-130, seed=8)
    _check(r)
    assert np.all(r["got"][0, 0, :130] == 0.0)


def test_v_scales_along_keys_reference_layout():
    _check(prefill_vs_oracle(1, 2, 1, 384, 384, 128, causal=True, v_axis=rk.V_SCALES_ALONG_KEYS, seed=9))
    _check(prefill_vs_oracle(1, 1, 1, 256, 200, 64, causal=False, v_axis=rk.V_SCALES_ALONG_KEYS, seed=10))


def test_e5m2_operands():
    for H in (2, 76):                                              # one item per CTA, and more
        _check(prefill_vs_oracle(1, H, 1, 256, 256, 128, causal=True, fmt=rk.E5M2, seed=11))


def test_mxfp6_operands_e2m3_q_e3m2_kv():
    """MXFP6 variant: E2M3 queries, E3M2 keys and values (P stays E4M3), 6-bit codes packed for the tensor core."""
    import oracle
    for (B, H, Hkv, Sq, Skv, d, axis) in ((1, 2, 1, 256, 256, 128, rk.V_SCALES_ALONG_D), (1, 4, 2, 200, 333, 64, rk.V_SCALES_ALONG_KEYS),
                                          (1, 76, 2, 256, 256, 128, rk.V_SCALES_ALONG_D), (2, 40, 2, 200, 333, 64, rk.V_SCALES_ALONG_KEYS),   # more items than CTAs
                                          (1, 2, 1, 384, 384, 256, rk.V_SCALES_ALONG_D)):
        Q, K, V = randn_qkv(B, H, Hkv, Sq, Skv, d, seed=31, mul=0.5)
        qc, qs = rk.mx_quantize(Q, rk.E2M3)
        kc, ks = rk.mx_quantize(K, rk.E3M2)
        vc, vs = rk.mx_quantize(V, rk.E3M2) if axis == rk.V_SCALES_ALONG_D else rk.mx_quantize_keys(V, rk.E3M2)
        o = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, softcap=50.0 if d == 256 else 0.0, q_fmt=rk.E2M3, kv_fmt=rk.E3M2,
                            v_scale_axis=axis)
        torch.cuda.synchronize()
        assert rk.last_device_status() == 0
        ref = oracle.attn_prefill(np_(qc), np_(kc), np_(vc), np_(qs), np_(ks), np_(vs), causal=True, softmax_scale=d ** -0.5,
                                  softcap=50.0 if d == 256 else 0.0, q_fmt=rk.E2M3, kv_fmt=rk.E3M2, v_scale_axis=axis, block_n=128)
        ma, rl = errors(np_(o.float()), ref["o_f32"])
        assert ma <= MAX_ABS and rl <= REL_L2, (d, ma, rl)
        for form in (PAIRS, TURNS, SPLIT) if d <= 128 else ():
            with prefill_form(form):
                assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, q_fmt=rk.E2M3, kv_fmt=rk.E3M2, v_scale_axis=axis), o), (H, form)
    assert rk.last_device_status() == 0


def test_mxfp4_operands_e2m1():
    """FP4 variant (lib/golden/mx_fp_math.h:238-246; the reference studies it in
    kernels/flash_attention_mx_gqa/fp6_attn_relerr.py:31-36): E2M1 queries, keys and values under E8M0 block scales,
    P stays E4M3; the 4-bit codes cross the interface one per byte and are packed two per byte for the tensor core.
    Also E2M1 keys/values under E4M3 queries, the mix a 4-bit KV cache gives."""
    import oracle
    for (B, H, Hkv, Sq, Skv, d, axis, qf) in ((1, 2, 1, 256, 256, 128, rk.V_SCALES_ALONG_D, rk.E2M1),
                                              (1, 4, 2, 200, 333, 64, rk.V_SCALES_ALONG_KEYS, rk.E2M1),
                                              (1, 2, 1, 384, 384, 256, rk.V_SCALES_ALONG_D, rk.E2M1),
                                              (2, 4, 2, 512, 512, 128, rk.V_SCALES_ALONG_KEYS, rk.E4M3)):
        Q, K, V = randn_qkv(B, H, Hkv, Sq, Skv, d, seed=37, mul=0.5)
        qc, qs = rk.mx_quantize(Q, qf)
        kc, ks = rk.mx_quantize(K, rk.E2M1)
        vc, vs = rk.mx_quantize(V, rk.E2M1) if axis == rk.V_SCALES_ALONG_D else rk.mx_quantize_keys(V, rk.E2M1)
        assert int(qc.max()) < (16 if qf == rk.E2M1 else 256) and int(kc.max()) < 16 and int(vc.max()) < 16
        o = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, softcap=50.0 if d == 256 else 0.0, q_fmt=qf, kv_fmt=rk.E2M1,
                            v_scale_axis=axis)
        torch.cuda.synchronize()
        assert rk.last_device_status() == 0
        ref = oracle.attn_prefill(np_(qc), np_(kc), np_(vc), np_(qs), np_(ks), np_(vs), causal=True, softmax_scale=d ** -0.5,
                                  softcap=50.0 if d == 256 else 0.0, q_fmt=qf, kv_fmt=rk.E2M1, v_scale_axis=axis, block_n=128)
        ma, rl = errors(np_(o.float()), ref["o_f32"])
        assert ma <= MAX_ABS and rl <= REL_L2, (d, ma, rl)


def test_dense_sub_byte_operands_give_the_same_output():
    """Operands handed over in the dense 6- / 4-bit form (rk_mx_pack_rows, rk_mx_pack_vt) -- what a KV cache kept in
    those formats holds -- give bit for bit the output of the call that packs them itself, and with scale-factor
    atoms on top the same again."""
    for (B, H, Hkv, Sq, Skv, d, qf, kvf, cap) in ((1, 4, 2, 200, 333, 64, rk.E2M3, rk.E3M2, 0.0),
                                                    (2, 4, 2, 512, 512, 128, rk.E2M1, rk.E2M1, 0.0),
                                                    (1, 2, 1, 384, 384, 256, rk.E2M3, rk.E3M2, 50.0)):
        Q, K, V = randn_qkv(B, H, Hkv, Sq, Skv, d, seed=41, mul=0.5)
        qc, qs = rk.mx_quantize(Q, qf)
        kc, ks = rk.mx_quantize(K, kvf)
        vc, vs = rk.mx_quantize_keys(V, kvf)
        want = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, softcap=cap, q_fmt=qf, kv_fmt=kvf,
                               v_scale_axis=rk.V_SCALES_ALONG_KEYS)
        qp, kp, vtp = rk.mx_pack_rows(qc, qf), rk.mx_pack_rows(kc, kvf), rk.mx_pack_vt(vc, kvf)
        bits_q, bits_kv = (4 if qf == rk.E2M1 else 6), (4 if kvf == rk.E2M1 else 6)
        dp, sp = (d + 127) // 128 * 128, (Skv + 127) // 128 * 128
        assert qp.shape == (B, H, Sq, dp * bits_q // 8) and kp.shape == (B, Hkv, Skv, dp * bits_kv // 8)
        assert vtp.shape == (B, Hkv, d, sp * bits_kv // 8)
        kw = dict(S_q=Sq, S_kv=Skv, d=d, q_fmt=qf, kv_fmt=kvf, causal=True, softcap=cap)
        got = rk.attn_prefill_packed(qp, kp, vtp, qs, ks, vs, **kw)
        assert torch.equal(got, want)
        # the first codes of a row, unpacked by hand
        row = qp[0, 0, 0].cpu().numpy().astype(np.uint64)
        word = int(row[0]) | int(row[1]) << 8 | int(row[2]) << 16
        first = [(word >> (bits_q * i)) & ((1 << bits_q) - 1) for i in range(3)]
        assert first == [int(x) for x in qc[0, 0, 0, :3].cpu()]
        # prepared all the way: scale-factor atoms as well, so that the call is the attention kernel alone
        _, qa = rk.mx_quantize_ex(Q, qf, rk.SCALES_SF_ATOMS)
        _, ka = rk.mx_quantize_ex(K, kvf, rk.SCALES_SF_ATOMS)
        _, va = rk.mx_quantize_keys_ex(V, kvf, rk.SCALES_SF_ATOMS)
        got2 = rk.attn_prefill_packed(qp, kp, vtp, qa, ka, va, q_scale_layout=rk.SCALES_SF_ATOMS,
                                      k_scale_layout=rk.SCALES_SF_ATOMS, v_scale_layout=rk.SCALES_SF_ATOMS, **kw)
        assert torch.equal(got2, want)
        torch.cuda.synchronize()
        assert rk.last_device_status() == 0
    # 8-bit formats have no dense form (the front end stops it; the library would answer RK_ERR_BAD_FORMAT)
    with pytest.raises((rk.RkError, ValueError)):
        rk.attn_prefill_packed(qp, kp, vtp, qs, ks, vs, S_q=Sq, S_kv=Skv, d=d, q_fmt=rk.E4M3, kv_fmt=rk.E3M2, causal=True)


@pytest.mark.parametrize("H", [1, 80])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("tile", [0, 1])
@pytest.mark.parametrize("softcap", [0.0, 50.0])
def test_a_key_tile_of_nan_scores_leaves_no_finite_row(H, d, tile, softcap):
    """E5M2 infinities in all columns of a key tile's K: every score of that tile is NaN, O is NaN and the log-sum-exp -inf (what a row sum
    that is not positive gives), whichever thread or group of threads had the tile."""
    qc, qs, kc, ks, vc, vs = quantize_inputs(*randn_qkv(1, H, H, 256, 256, d, seed=64), fmt=rk.E5M2)
    kc[:, :, tile * 128:(tile + 1) * 128] = 0x7C
    for form in (0, PAIRS, TURNS, SPLIT) if d <= 128 else (0,):
        lse = torch.zeros(1, H, 256, device="cuda")
        with prefill_form(form):
            o = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=False, softcap=softcap, lse=lse, q_fmt=rk.E5M2, kv_fmt=rk.E5M2)
        assert torch.isnan(o).all() and torch.isneginf(lse).all(), form
    assert rk.last_device_status() == 0


def test_lse_output():
    r = prefill_vs_oracle(1, 2, 1, 256, 256, 128, causal=True, want_lse=True, seed=12)
    _check(r)
    assert np.abs(r["lse"] - r["ref"]["lse"]).max() < 1e-3


@pytest.mark.parametrize("B,H,Hkv,S,d,causal,form", [
    (2, 4, 2, 1024, 128, True, 0),
    (8, 64, 64, 200, 64, False, PAIRS), (8, 64, 64, 160, 128, False, PAIRS),      # the second query tile of every pair ends inside its TMEM lane quadrants
    (8, 64, 64, 200, 64, False, TURNS), (8, 64, 64, 160, 128, False, TURNS),
    (2, 20, 10, 640, 256, False, 0)])                               # 200 query tiles of five key tiles
def test_bit_identical_across_runs(B, H, Hkv, S, d, causal, form):
    """Race check borrowed from the reference ("bit-identical O across 13 runs",
    kernels/flash_attention_mx/kernel.cpp:158-160)."""
    Q, K, V = randn_qkv(B, H, Hkv, S, S, d, seed=13)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    with prefill_form(form):
        first = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=causal)
        for _ in range(5):
            again = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=causal)
            assert torch.equal(first, again)
    assert rk.last_device_status() == 0


def test_host_buffer_entry_point_matches_device_one():
    Q, K, V = randn_qkv(1, 4, 2, 512, 512, 128, seed=14)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    dev = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True)
    host = rk.attn_prefill_host(*[t.cpu().pin_memory() for t in (qc, kc, vc, qs, ks, vs)], causal=True)
    assert torch.equal(dev.cpu(), host)


@pytest.mark.parametrize("B,H,Hkv,S,axis", [(3, 6, 3, 256, 1), (10, 2, 2, 128, 0), (2, 8, 8, 160, 1), (9, 4, 1, 128, 1)])
def test_host_entry_point_chunking(B, H, Hkv, S, axis):
    """The host entry point cuts the call into chunks of whole (batch, KV head) units (ranges of KV heads when
    the batch is small, groups of batches when it is large): every chunking gives the device call's bits, for O
    and for the log-sum-exp, with either V scale layout and a ragged sequence length."""
    Q, K, V = randn_qkv(B, H, Hkv, S, S, 128, seed=40 + B)
    qc, qs = rk.mx_quantize(Q); kc, ks = rk.mx_quantize(K)
    vc, vs = rk.mx_quantize(V) if axis == 1 else rk.mx_quantize_keys(V)
    lse = torch.empty(B, H, S, dtype=torch.float32, device="cuda")
    dev = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, v_scale_axis=axis, lse=lse)
    runner = rk.PrefillHostRunner(*[t.cpu().pin_memory() for t in (qc, kc, vc, qs, ks, vs)], causal=True,
                                  v_scale_axis=axis, want_lse=True)
    for _ in range(2):                      # twice: the shared copy streams and events are reused
        host = runner.run()
        assert torch.equal(dev.cpu(), host)
        assert torch.equal(lse.cpu(), runner.lse)
    assert rk.last_device_status() == 0


def test_full_size_head_slices_match_oracle():
    """B=8 H=16 S=4096 d=128 causal (the benchmark workload): the whole tensor runs on the GPU, two
    (batch, head) slices are checked against the oracle, and every row is checked for the size-independent
    property that O is a convex combination of V rows (|O| <= max|V| per column block)."""
    B, H, S, d = 8, 16, 4096, 128
    Q, K, V = randn_qkv(B, H, H, S, S, d, seed=15)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    del Q, K
    o = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    assert torch.isfinite(o.float()).all()
    assert o.float().abs().max() <= V.abs().max() * 1.01
    for sl in (0, B * H - 1):
        b, h = divmod(sl, H)
        ref = oracle.attn_prefill(np_(qc[b:b + 1, h:h + 1]), np_(kc[b:b + 1, h:h + 1]), np_(vc[b:b + 1, h:h + 1]),
                                  np_(qs[b:b + 1, h:h + 1]), np_(ks[b:b + 1, h:h + 1]), np_(vs[b:b + 1, h:h + 1]),
                                  causal=True, softmax_scale=d ** -0.5, block_n=128)
        ma, rl = errors(np_(o[b, h].float()), ref["o_f32"][0, 0])
        assert ma <= MAX_ABS and rl <= REL_L2, (sl, ma, rl)


@pytest.mark.parametrize("form", [PAIRS, TURNS, SPLIT])
@pytest.mark.parametrize("d,qmul,H", [(128, 1.0, 1), (128, 6.0, 1), (64, 1.0, 1), (128, 1.0, 75), (128, 6.0, 75), (64, 1.0, 75)])
def test_stage_parity_s_and_requantized_p(d, qmul, H, form):
    """Stage-level parity on the first key tile of the last query tile of head 0 (the kernels' debug dump), in every form, with one item per
    CTA (one head) and more (75): S = Q K^T within
    fp32 reassociation error, and the requantized P -- E4M3 codes and E8M0 block scales -- equal to the oracle's.
    A code may differ by one step where the fp32 p sits on a truncation boundary; such elements are counted and
    must stay below 0.05 %."""
    import ctypes as C
    Sq = Skv = 256
    Q, K, V = randn_qkv(1, H, H, Sq, Skv, d, seed=50, qmul=qmul)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    dbg = torch.zeros(32768, dtype=torch.float32, device="cuda")
    rk.lib().rk_debug_set_prefill_dump(C.c_void_p(dbg.data_ptr()))
    try:
        with prefill_form(form):
            rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True)
        torch.cuda.synchronize()
    finally:
        rk.lib().rk_debug_set_prefill_dump(None)
    assert rk.last_device_status() == 0
    scale = d ** -0.5
    r = oracle.attn_prefill(*(np_(t[:, :1]) for t in (qc, kc, vc, qs, ks, vs)), causal=True, softmax_scale=scale,
                            block_n=128, dump_slice=0)
    dd = np_(dbg)
    rows = slice(128, 256)                                    # the dump is the last query tile, key tile 0
    s_gpu = dd[:128 * 128].reshape(128, 128)
    s_ref = r["s"][rows, :128] / scale
    assert np.abs(s_gpu - s_ref).max() <= 1e-5 * np.abs(s_ref).max() + 1e-6
    pcodes = dd[128 * 128: 128 * 128 + 128 * 32].view(np.uint8).reshape(128, 128)
    pscale = dd[128 * 128 + 128 * 32: 128 * 128 + 128 * 32 + 128].view(np.uint8).reshape(128, 4)
    assert np.array_equal(pscale, r["p_scales"][rows, :4])
    diff = pcodes.astype(np.int32) - r["p_codes"][rows, :128].astype(np.int32)
    bad = np.count_nonzero(diff)
    assert np.abs(diff).max() <= 1 and bad <= 0.0005 * diff.size, (bad, int(np.abs(diff).max()))
    # running max and row sum after the tile's last key tile: m is kept in the log2 domain on the GPU
    ml = dd[128 * 128 + 128 * 32 + 128: 128 * 128 + 128 * 32 + 128 + 256].reshape(128, 2)
    m_gpu, l_gpu = ml[:, 0] * np.log(2.0), ml[:, 1]
    assert np.abs(m_gpu - r["m"][rows]).max() <= 4e-6 * np.abs(r["m"][rows]).max() + 1e-6
    assert np.abs(l_gpu / r["l"][rows] - 1.0).max() <= 1e-4


@pytest.mark.parametrize("B,H,Hkv,Sq,Skv,d,kw", [
    (1, 148, 4, 33, 160, 128, dict(causal=False)),                # 148 query tiles: one for every SM, a CTA each
    (1, 149, 149, 33, 160, 128, dict(causal=False)),              # one more: a CTA takes two, here one that exists
    (1, 50, 10, 300, 300, 64, dict(causal=True)),                 # three tiles of a head: the last pair has one
    (3, 17, 17, 257, 257, 128, dict(causal=True, window=140)),
    (2, 40, 8, 256, 400, 128, dict(causal=True, q_pos0=144, softcap=5.0)),
    (1, 4, 4, 509, 700, 128, dict(causal=True, q_pos0=191, window=130, softcap=5.0)),
    (1, 2, 1, 1, 129, 128, dict(causal=True, q_pos0=128)),        # one query, one key in the last key tile
    (1, 2, 2, 130, 65, 64, dict(causal=True))])                   # keys of one half of a key tile, and one of the other
def test_grids_on_both_sides_of_one_query_tile_per_sm(B, H, Hkv, Sq, Skv, d, kw):
    """Grids of no more query tiles than SMs and of a few more; odd numbers of tiles, masks that cut a key tile in either half."""
    _check(prefill_vs_oracle(B, H, Hkv, Sq, Skv, d, seed=61, **kw))


@pytest.mark.parametrize("B,H,Hkv,Sq,Skv,d,kw", [
    (1, 4, 2, 130, 513, 128, dict(causal=True, q_pos0=383)),      # one item per CTA, five key tiles, the last of one key
    (2, 59, 59, 260, 260, 128, dict(causal=True)),                # three items of 1, 2, 3 key tiles per head, 354 in all: a CTA's items start on either group
    (1, 350, 7, 40, 100, 64, dict(causal=False)),                 # items of one key tile one after the other
    (1, 88, 8, 390, 390, 64, dict(causal=True, q_pos0=-130)),     # items without a key tile between others
    (1, 58, 2, 700, 700, 128, dict(causal=True, window=150)),     # windows: masks at both ends of an item's key tiles
    (1, 80, 8, 500, 500, 128, dict(causal=True, softcap=5.0)),    # the mask in registers
    (1, 16, 4, 1100, 1100, 128, dict(causal=True))])
def test_query_tiles_one_after_the_other_with_key_tiles_in_turn(B, H, Hkv, Sq, Skv, d, kw):
    """Calls of few query tiles: a CTA has one at a time, its softmax groups take the key tiles in turn."""
    _check(prefill_vs_oracle(B, H, Hkv, Sq, Skv, d, seed=63, **kw))


@pytest.mark.parametrize("fmt", [rk.E4M3, rk.E5M2, rk.E2M3, rk.E3M2, rk.E2M1])
@pytest.mark.parametrize("S,d", [(31, 64), (129, 64), (333, 128), (160, 256)])
def test_v_preparation_equals_the_oracle_re_blocking(S, d, fmt):
    """V with scales along d, re-blocked (and for 6- and 4-bit codes packed and transposed) by the call, against the same V
    re-blocked by the oracle and handed over with scales along the keys: bit for bit the same output, because the attention
    kernel then reads the same operands.  Row scales that span 2^50 inside a block take the slow form."""
    rng = np.random.default_rng(71 + fmt)
    Q, K, V = randn_qkv(1, 3, 3, 140, S, d, seed=73)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V, fmt=fmt)
    vs[0, 0] = torch.from_numpy(rng.integers(80, 131, size=(S, d // 32), dtype=np.uint8)).cuda()
    vs[0, 1] = torch.from_numpy(rng.integers(122, 131, size=(S, d // 32), dtype=np.uint8)).cuda()
    pairs = [oracle.rebase_v(np_(vc[0, h]), np_(vs[0, h]), fmt) for h in range(3)]
    rc, rs = (torch.from_numpy(np.stack([x[i] for x in pairs])[None]).cuda() for i in range(2))
    kw = dict(causal=False, q_fmt=fmt, kv_fmt=fmt)
    got = rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
    want = rk.attn_prefill(qc, kc, rc, qs, ks, rs, v_scale_axis=rk.V_SCALES_ALONG_KEYS, **kw)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    assert torch.isfinite(want.float()).all() and torch.equal(got, want)


@pytest.mark.parametrize("B,H,Hkv,S,d,kw", [
    (1, 16, 16, 2048, 128, dict(causal=True)),                    # 256 query tiles: one at a time, also in the pieces
    (1, 32, 32, 2048, 128, dict(causal=True)),                    # 512: pairs, and the pieces one at a time
    (2, 32, 16, 1090, 64, dict(causal=True, window=300)),         # 576, odd numbers of tiles per head: the same
    (8, 18, 9, 512, 64, dict(causal=False)),                      # 576 of equal length: the same
    (1, 40, 10, 500, 128, dict(causal=True, softcap=5.0)),        # 160: one at a time, the pieces with both groups on every key tile
    (1, 40, 10, 500, 128, dict(causal=False, softcap=5.0)),       # pairs, the pieces with both groups on every key tile
    (2, 12, 4, 1090, 64, dict(causal=True, window=300)),
    (2, 100, 50, 200, 64, dict(causal=False)),                    # lane quadrants that have no row
    (2, 90, 90, 140, 128, dict(causal=False)),
    (1, 20, 10, 1200, 128, dict(causal=True)),
    (2, 20, 10, 640, 256, dict(causal=False)),                    # 200 of five key tiles: a CTA's second item starts on an odd one
    (2, 20, 10, 640, 256, dict(causal=True, softcap=50.0)),       # items of one key tile at the end of the work order, one after the other
    (6, 100, 50, 100, 256, dict(causal=True)),                    # 600 items of one key tile
    (2, 100, 100, 128, 256, dict(causal=False, softcap=50.0))])
def test_smaller_calls_give_the_same_bits_on_both_sides_of_one_query_tile_per_sm(B, H, Hkv, S, d, kw):
    """A call whose query tiles outnumber the SMs, against the same call cut by the host entry point and unit by unit, where each
    piece has a CTA per tile: O and the log-sum-exp are equal bit for bit (the row sum is taken in one order in every form, and at d = 256
    whatever the CTA worked on before).  At d <= 128 the whole call in the other forms too."""
    Q, K, V = randn_qkv(B, H, Hkv, S, S, d, seed=62)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    lse = torch.empty(B, H, S, dtype=torch.float32, device="cuda")
    o = rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=lse, **kw)
    for form in (PAIRS, TURNS, SPLIT) if d <= 128 else ():
        with prefill_form(form):
            l1 = torch.empty_like(lse)
            assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=l1, **kw), o) and torch.equal(l1, lse), form
    sms, grp = torch.cuda.get_device_properties(0).multi_processor_count, H // Hkv
    assert B * H * ((S + 127) // 128) > sms >= grp * ((S + 127) // 128)
    for b in range(B):
        for h in range(Hkv):
            part = [t[b:b + 1, h * grp:(h + 1) * grp].contiguous() for t in (qc, qs)] + [t[b:b + 1, h:h + 1].contiguous() for t in (kc, ks, vc, vs)]
            l1 = torch.empty(1, grp, S, dtype=torch.float32, device="cuda")
            o1 = rk.attn_prefill(part[0], part[2], part[4], part[1], part[3], part[5], lse=l1, **kw)
            assert torch.equal(o1[0], o[b, h * grp:(h + 1) * grp]) and torch.equal(l1[0], lse[b, h * grp:(h + 1) * grp]), (b, h)
    runner = rk.PrefillHostRunner(*[t.cpu().pin_memory() for t in (qc, kc, vc, qs, ks, vs)], want_lse=True, **kw)
    assert torch.equal(runner.run(), o.cpu()) and torch.equal(runner.lse, lse.cpu())
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("B,H,Hkv,S,d,kw,whole,piece", [
    (1, 32, 32, 2048, 128, dict(causal=True), PAIRS, TURNS), (2, 32, 16, 1090, 64, dict(causal=True, window=300), PAIRS, TURNS),
    (8, 18, 9, 512, 64, dict(causal=False), PAIRS, TURNS), (1, 40, 10, 500, 128, dict(causal=True, softcap=5.0), TURNS, SPLIT),
    (1, 40, 10, 500, 128, dict(causal=False, softcap=5.0), PAIRS, SPLIT), (2, 100, 50, 200, 64, dict(causal=False), TURNS, SPLIT)])
def test_forms_of_a_call_and_of_its_pieces(B, H, Hkv, S, d, kw, whole, piece):
    """The test above sees every pair of forms that a call and its pieces can have (148 SMs)."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shapes are chosen for 148 SMs")
    assert chosen_form(B, H, S, S, d, **kw) == whole and chosen_form(1, H // Hkv, S, S, d, **kw) == piece


@pytest.mark.parametrize("key,factor", [(5, 20.0), (5, 30.0), (70, 20.0), (70, 30.0)])
def test_smaller_calls_give_the_same_bits_around_the_soft_caps_series_limit(key, factor):
    """One key of every key tile has logits on both sides of cap / 8, the others far below: the exponential form of the cap for that key's
    half of the tile and the series for the other, in every form and with a CTA per tile."""
    Q, K, V = randn_qkv(1, 40, 10, 500, 500, 128, seed=63, mul=0.3)
    K[:, :, key::128] *= factor                                   # logits of standard deviation 1.8 and 2.7, 128 rows x 4 tiles of them a head
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    kw = dict(causal=False, softcap=50.0)
    lse = torch.empty(1, 40, 500, dtype=torch.float32, device="cuda")
    o = rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=lse, **kw)
    for form in (PAIRS, TURNS, SPLIT):
        with prefill_form(form):
            l1 = torch.empty_like(lse)
            assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=l1, **kw), o) and torch.equal(l1, lse), form
    for h in range(10):
        part = [t[:, h * 4:(h + 1) * 4].contiguous() for t in (qc, qs)] + [t[:, h:h + 1].contiguous() for t in (kc, ks, vc, vs)]
        l1 = torch.empty(1, 4, 500, dtype=torch.float32, device="cuda")
        o1 = rk.attn_prefill(part[0], part[2], part[4], part[1], part[3], part[5], lse=l1, **kw)
        assert torch.equal(o1[0], o[0, h * 4:(h + 1) * 4]) and torch.equal(l1[0], lse[0, h * 4:(h + 1) * 4]), h
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("B,H,Hkv,Sq,Skv,d,kw", [
    (5, 64, 32, 300, 300, 128, dict(causal=True)),                   # 640 pairs, every second without its second tile; two tiles at most
    (3, 64, 32, 129, 389, 128, dict(causal=False)),                  # one key in the last tile, equal numbers of key tiles
    (4, 48, 48, 520, 520, 64, dict(causal=True, window=129)),        # items that start inside the sequence
    (2, 96, 96, 200, 200, 128, dict(causal=True, q_pos0=-130)),      # a tile without a visible key before one that has some
    (2, 100, 50, 260, 390, 128, dict(causal=True, q_pos0=130, softcap=5.0)),
    (3, 60, 20, 260, 260, 256, dict(causal=True)),                   # 540 items of one, two and three key tiles
    (2, 80, 80, 140, 400, 256, dict(causal=False, softcap=50.0)),
    (2, 90, 45, 200, 200, 256, dict(causal=True, q_pos0=-130, softcap=50.0)),
    (1, 80, 80, 390, 390, 256, dict(causal=True, window=128)),
])
def test_many_items_per_sm(B, H, Hkv, Sq, Skv, d, kw):
    """A CTA takes one item after the other: odd and even numbers of key tiles, items without one, the last O written out at the end."""
    r = prefill_vs_oracle(B, H, Hkv, Sq, Skv, d, seed=31, want_lse=True, **kw)
    # Millions of rows, some of few keys: beyond the general bound the bf16 rounding of |O| up to 5 (2^-8 |O|), and, where exp2 of the two sides
    # falls on either side of a code boundary, one E4M3 step of a P, 2^-3 of its weight: 2^-3 * 0.1 * 4.5 for the largest |v|.
    assert r["err"][1] <= REL_L2 and (np.abs(r["got"] - r["ref"]["o_f32"]) <= 0.056 + 2.0 ** -8 * np.abs(r["ref"]["o_f32"])).all(), r["err"]
    seen = np.isfinite(r["ref"]["lse"])
    assert (np.isfinite(r["lse"]) == seen).all() and np.abs(r["lse"][seen] - r["ref"]["lse"][seen]).max() <= 1e-3


@pytest.mark.parametrize("d,window", [(128, 1), (128, 127), (128, 128), (128, 129), (64, 256), (64, 257), (256, 127), (256, 129)])
def test_window_edges_against_tile_edges(d, window):
    _check(prefill_vs_oracle(2, 4, 2, 515, 600, d, causal=True, q_pos0=85, window=window, seed=32))


@pytest.mark.parametrize("H,Sq,d,form", [(2, 150, 64, SPLIT), (2, 150, 128, SPLIT), (160, 150, 128, PAIRS), (160, 150, 128, TURNS), (2, 150, 64, TURNS), (2, 150, 256, 0)])
def test_o_at_a_16_byte_boundary(H, Sq, d, form):
    """O need not be 32-byte aligned: rows then leave in 16-byte stores.  The same bits, nothing beside them."""
    q, qs, k, ks, v, vs = quantize_inputs(*randn_qkv(1, H, H, Sq, Sq, d, 33))
    want = rk.attn_prefill(q, k, v, qs, ks, vs, causal=True)
    flat = torch.full((want.numel() + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
    out = flat[8:8 + want.numel()].view(want.shape)
    assert out.data_ptr() % 32 == 16
    with prefill_form(form):
        rk.attn_prefill(q, k, v, qs, ks, vs, causal=True, out=out)
    assert torch.equal(out, want) and (flat[:8] == 7.0).all() and (flat[-8:] == 7.0).all()


@pytest.mark.parametrize("H,Sq,Skv,d,causal,q_pos0", [(2, 300, 300, 128, False, 0), (160, 200, 333, 64, False, -130), (200, 520, 700, 128, False, -130),
                                                     (2, 300, 300, 256, False, -130), (2, 300, 300, 128, True, 0)])
@pytest.mark.parametrize("beyond", [True, False])
def test_windows_that_mask_nothing_or_little(H, Sq, Skv, d, causal, q_pos0, beyond):
    """A window near 2^31, a caller's "no limit", masks no key: the bits of a call without one.  The largest window that masks one, the first key for the last
    row alone: the bits of that call in every other row."""
    qc, qs, kc, ks, vc, vs = quantize_inputs(*randn_qkv(1, H, H, Sq, Skv, d, seed=34))
    kw = dict(causal=causal, q_pos0=q_pos0)
    want = rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
    last = q_pos0 + Sq - 1
    for window in ((2 ** 31 - 1, 2 ** 31 - 100, last + 1) if beyond else (last,)):
        got = rk.attn_prefill(qc, kc, vc, qs, ks, vs, window=window, **kw)
        assert torch.equal(got[:, :, :-1], want[:, :, :-1]) and torch.equal(got[:, :, -1], want[:, :, -1]) == beyond, window
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("S_q,S_kv,d,fmt,kw", [(1, 1, 128, 0, {}), (17, 31, 64, 0, {}), (128, 128, 128, 0, {}), (129, 129, 64, 1, {}), (40, 33, 128, 0, dict(causal=False)), (200, 256, 128, 1, dict(q_pos0=56)),
                                               (256, 256, 64, 0, dict(causal=False)), (7, 257, 64, 0, dict(q_pos0=250)), (300, 383, 128, 0, dict(q_pos0=83, window=100)), (130, 384, 64, 1, dict(causal=False)),
                                               (384, 384, 128, 0, {}), (64, 128, 128, 0, dict(q_pos0=-70))])
@pytest.mark.parametrize("hard", [False, True])
def test_calls_that_prepare_their_operands_themselves(S_q, S_kv, d, fmt, kw, hard):
    """Calls of up to three key tiles re-block V and order the scales inside the attention kernel: the same bits as by pairs of query tiles, which have the preparation launch, V scaled along d or along the keys. Edges of key
    blocks and tiles, scales at odd addresses; hard: V of any code, zeros and subnormals, under scales that are close, far apart or extreme."""
    B, H, H_kv = 2, 16, 8
    g = torch.Generator(device="cuda").manual_seed(S_q + S_kv + d)
    def odd(t):
        flat = torch.empty(t.numel() + 1, dtype=torch.uint8, device="cuda")
        flat[1:] = t.flatten()
        return flat[1:].view(t.shape)
    q, qs = rk.mx_quantize(torch.randn(B, H, S_q, d, generator=g, device="cuda"), fmt)
    k, ks = rk.mx_quantize(torch.randn(B, H_kv, S_kv, d, generator=g, device="cuda"), fmt)
    v, vs = rk.mx_quantize(torch.randn(B, H_kv, S_kv, d, generator=g, device="cuda"), fmt)
    if hard:
        v = torch.randint(0, 256, v.shape, generator=g, device="cuda", dtype=torch.uint8)
        v[(v & 0x7F) >= (0x7F if fmt == 0 else 0x7C)] = 0x38
        v[0, 0, :, :4] = 0
        v[0, 1] &= 0x87 if fmt == 0 else 0x83
        vs = torch.randint(118, 130, vs.shape, generator=g, device="cuda", dtype=torch.uint8)
        vs[1, 0] = torch.randint(90, 140, vs[1, 0].shape, generator=g, device="cuda", dtype=torch.uint8)
        vs[1, 1] = torch.randint(1, 30, vs[1, 1].shape, generator=g, device="cuda", dtype=torch.uint8)
    kw = dict(dict(causal=True), **kw)
    vr, vrs = rk.mx_rebase_v(v, vs, fmt)
    lse = [torch.full((B, H, S_q), 7.0, device="cuda") for _ in range(2)]
    along_keys = dict(v_scale_axis=rk.V_SCALES_ALONG_KEYS)
    with prefill_form(PAIRS):
        want = rk.attn_prefill(q, k, vr, qs, ks, vrs, q_fmt=fmt, kv_fmt=fmt, lse=lse[0], **along_keys, **kw)
    for shift in (lambda t: t, odd):
        for axis, codes, scales in (({}, v, vs), (along_keys, vr, vrs)):
            lse[1].fill_(7.0)
            got = rk.attn_prefill(q, k, codes, shift(qs), shift(ks), shift(scales), q_fmt=fmt, kv_fmt=fmt, lse=lse[1], **axis, **kw)
            assert torch.equal(got.view(torch.int16), want.view(torch.int16))
            assert torch.equal(lse[1], lse[0])
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("S_q,S_kv,d,fmt", [(130, 700, 64, rk.E4M3), (257, 513, 64, rk.E2M3), (33, 640, 128, rk.E4M3), (300, 600, 256, rk.E4M3), (140, 200, 256, rk.E2M1)])
def test_scales_at_any_address(S_q, S_kv, d, fmt):
    """Row-major scales of calls with a preparation launch, read as words, halves or bytes: the same bits from every address, ragged tiles among them."""
    g = torch.Generator(device="cuda").manual_seed(S_q + d)
    q, qs = rk.mx_quantize(torch.randn(2, 4, S_q, d, generator=g, device="cuda"), fmt)
    k, ks = rk.mx_quantize(torch.randn(2, 2, S_kv, d, generator=g, device="cuda"), fmt)
    v, vs = rk.mx_quantize(torch.randn(2, 2, S_kv, d, generator=g, device="cuda"), fmt)
    def moved(t, n):
        flat = torch.full((t.numel() + n + 256,), 0xFE, dtype=torch.uint8, device="cuda")
        flat[n:n + t.numel()] = t.flatten()
        return flat[n:n + t.numel()].view(t.shape)
    kw = dict(causal=True, q_pos0=S_kv - S_q, q_fmt=fmt, kv_fmt=fmt)
    with prefill_form(PAIRS):
        want = rk.attn_prefill(q, k, v, qs, ks, vs, **kw)
        for n in (1, 2, 3):
            assert torch.equal(rk.attn_prefill(q, k, v, moved(qs, n), moved(ks, n), moved(vs, n), **kw), want), n
    assert rk.last_device_status() == 0
