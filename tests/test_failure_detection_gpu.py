"""Failure detection without a GPU fault: a bounded device-side wait is made to run out (an mbarrier nobody ever
arrives at, limit one millisecond) and the library must report it, keep later launches from producing results
while the status word is set, and work again once the word has been read.  Plus the schedule-perturbation check
the reference uses to hunt missing barriers (a delay in one role must not change a bit of O:
kernels/flash_attention_mx_stable/README.md:27-35)."""
import ctypes as C

import pytest
import torch

import radiance_kernels_b200 as rk
from radiance_kernels_b200._lib import DecodeArgs, PrefillArgs
from helpers import PAIRS, SPLIT, TURNS, prefill_form, quantize_inputs, randn_qkv

pytestmark = pytest.mark.gpu

WAIT_GAVE_UP = 901          # the code the test-hook kernel records


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def test_bounded_wait_runs_out_and_is_reported_and_clears():
    L = rk.lib()
    assert rk.last_device_status() == 0
    Q, K, V = randn_qkv(1, 2, 2, 256, 256, 128, seed=90)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    good = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True)
    torch.cuda.synchronize()

    assert L.rk_debug_wait_runs_out(1000, 0, _stream()) == 0            # the kernel returns by itself
    torch.cuda.synchronize()
    try:
        # while the word is set, launches return at once and write nothing
        sentinel = torch.full_like(good, 7.0)
        out = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, out=sentinel.clone())
        torch.cuda.synchronize()
        assert torch.equal(out, sentinel)
        status = rk.last_device_status()
    except BaseException:
        rk.last_device_status()                                         # never leave the word set for the tests that follow
        raise
    assert status == WAIT_GAVE_UP                                       # reported once ...
    assert rk.last_device_status() == 0                                 # ... and cleared by the read
    again = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True)
    torch.cuda.synchronize()
    assert torch.equal(again, good)
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("longer", [0, 1])
def test_waits_bounded_by_polls_run_out_after_about_two_seconds(longer):
    """The waits of the prefill kernels that count polls instead of time, with 1/64 of the polls: they run out, and 64 times that lies between half a second
    and five.  The CTA's abort flag ends them at once."""
    L = rk.lib()
    assert rk.last_device_status() == 0
    for aborted in (0, 1):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        assert L.rk_debug_compact_wait_runs_out(longer, aborted, _stream()) == 0
        e1.record()
        torch.cuda.synchronize()
        assert rk.last_device_status() == 902 + longer
        seconds = e0.elapsed_time(e1) * 64 / 1000
        assert seconds < 0.02 if aborted else 0.5 < seconds < 5.0, (aborted, seconds)


@pytest.mark.parametrize("H,S,d,q_pos0,form", [(2, 300, 256, 0, 0), (160, 200, 256, -130, 0), (160, 100, 128, 0, TURNS), (160, 200, 64, -130, TURNS),
                                               (300, 300, 128, 0, PAIRS), (300, 200, 64, -130, PAIRS), (2, 300, 128, 0, SPLIT), (60, 200, 64, -130, SPLIT)])
def test_prefill_writes_nothing_while_the_status_word_is_set(H, S, d, q_pos0, form):
    """Every form of the prefill kernels, items of one key tile and query tiles without a visible key among them: neither O nor the
    log-sum-exps are touched."""
    L = rk.lib()
    qc, qs, kc, ks, vc, vs = quantize_inputs(*randn_qkv(1, H, H, S, S, d, seed=92))
    o = torch.full((1, H, S, d), 7.0, dtype=torch.bfloat16, device="cuda")
    lse = torch.full((1, H, S), 7.0, device="cuda")
    assert rk.last_device_status() == 0
    assert L.rk_debug_wait_runs_out(1000, 0, _stream()) == 0
    torch.cuda.synchronize()
    try:
        with prefill_form(form):
            rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, q_pos0=q_pos0, out=o, lse=lse)
        torch.cuda.synchronize()
    finally:
        status = rk.last_device_status()
    assert status == WAIT_GAVE_UP and (o == 7.0).all() and (lse == 7.0).all()
    with prefill_form(form):
        rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=True, q_pos0=q_pos0, out=o, lse=lse)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0 and not (o == 7.0).all() and not (lse == 7.0).any()


@pytest.mark.parametrize("H,S,d,form", [(2, 600, 128, TURNS), (100, 600, 128, TURNS), (200, 300, 64, TURNS), (2, 300, 128, SPLIT), (30, 600, 64, SPLIT),
                                        (2, 600, 128, PAIRS), (300, 512, 128, PAIRS), (250, 1024, 64, PAIRS), (2, 600, 256, 0), (100, 600, 256, 0)])
def test_a_role_that_gives_up_ends_the_call_and_the_next_one_is_whole(H, S, d, form):
    """One warp role at a time (either softmax group, correction, TMA producer, Q K^T and P V issuer) acts after a key tile as if its
    wait had run out: loads, MMAs and stores are under way, the other roles see the CTA's flag, the kernel ends, a code is reported and the next
    call has every bit of the one before.  At d <= 128 in every form, one item per CTA and many."""
    L = rk.lib()
    qc, qs, kc, ks, vc, vs = quantize_inputs(*randn_qkv(1, H, H, S, S, d, seed=93))
    with prefill_form(form):
        want = rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=False)
        assert rk.last_device_status() == 0
        for role in (1, 2, 3, 4, 5, 6):
            if d == 256 and role == 3:
                continue                                                # no correction warps there
            L.rk_debug_set_prefill_perturb(100 + role)
            try:
                rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=False)
                torch.cuda.synchronize()
            finally:
                L.rk_debug_set_prefill_perturb(0)
                status = rk.last_device_status()
            assert 100 < status < 600, (role, status)
            assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, causal=False), want), role
            assert rk.last_device_status() == 0


@pytest.mark.parametrize("kernel,role,code", [("rmsnorm", 1, 602), ("rmsnorm", 2, 602), ("rope", 1, 601)])
def test_a_ring_of_copies_that_gives_up_ends_the_call_and_the_next_one_is_whole(kernel, role, code):
    """The RoPE and RMSNorm kernels that read by bulk copies: the readers, or the warp that asks for the copies, act after a few of them as if their wait had
    run out, with others under way.  The kernel waits for those, reports a code (RMSNorm: without a byte written), and the next calls have every bit."""
    L = rk.lib()
    g = torch.Generator(device="cuda").manual_seed(95)
    if kernel == "rmsnorm":
        x, gamma = torch.randn(1200, 4096, generator=g, device="cuda").bfloat16(), torch.rand(4096, generator=g, device="cuda") + 0.5
        call = lambda: rk.rmsnorm_mx_quantize(x, gamma, 1e-5)
    else:
        S, d = 4096, 128
        x = torch.randn(1, 32, S, d, generator=g, device="cuda")
        ang = torch.rand(S, d // 2, generator=g, device="cuda")
        cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
        assert L.rk_debug_rope_by_copies(32 * S, d, S, torch.cuda.get_device_properties(0).multi_processor_count)
        call = lambda: rk.rope_mx_quantize(x, cos, sin)
    want = call()
    assert rk.last_device_status() == 0
    L.rk_debug_set_ring_stop(role)
    try:
        call()
        torch.cuda.synchronize()
    finally:
        L.rk_debug_set_ring_stop(0)
        status = rk.last_device_status()
    assert status == code
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(call(), want))
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("role", [1, 2])
def test_the_ring_of_a_large_rmsnorm_call_that_gives_up(role):
    """The same for RMSNorm calls of more rows than lie on the chip at once (the test above has fewer, which come in one copy each)."""
    L = rk.lib()
    g = torch.Generator(device="cuda").manual_seed(96)
    x, gamma = torch.randn(4500, 4096, generator=g, device="cuda").bfloat16(), torch.rand(4096, generator=g, device="cuda") + 0.5
    want = rk.rmsnorm_mx_quantize(x, gamma, 1e-5)
    L.rk_debug_set_ring_stop(role)
    try:
        rk.rmsnorm_mx_quantize(x, gamma, 1e-5)
        torch.cuda.synchronize()
    finally:
        L.rk_debug_set_ring_stop(0)
        status = rk.last_device_status()
    assert status == 602
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(rk.rmsnorm_mx_quantize(x, gamma, 1e-5), want))
    assert rk.last_device_status() == 0


def test_noalloc_decode_status_word_is_observable():
    L = rk.lib()
    g = torch.Generator(device="cuda").manual_seed(91)
    q = torch.randn(1, 8, 128, generator=g, device="cuda").bfloat16()
    kc, ks = rk.mx_quantize(torch.randn(1, 2, 512, 128, generator=g, device="cuda"))
    vc, vs = rk.mx_quantize(torch.randn(1, 2, 512, 128, generator=g, device="cuda"))
    want = rk.attn_decode(q, kc, vc, ks, vs)

    def call():
        o = torch.zeros(1, 8, 128, dtype=torch.bfloat16, device="cuda")
        a = DecodeArgs()
        a.q, a.k, a.v, a.k_scale, a.v_scale = (C.c_void_p(t.data_ptr()) for t in (q, kc, vc, ks, vs))
        a.o = C.c_void_p(o.data_ptr())
        a.B, a.H, a.H_kv, a.L, a.d = 1, 8, 2, 512, 128
        assert L.rk_attn_decode_noalloc(C.byref(a), _stream()) == 0
        torch.cuda.synchronize()
        return o

    assert L.rk_attn_decode_noalloc_status() == 0
    assert L.rk_debug_wait_runs_out(1000, 1, _stream()) == 0
    call()                                                              # runs on a set word: its result is not valid
    assert L.rk_attn_decode_noalloc_status() == WAIT_GAVE_UP
    assert rk.last_device_status() == 0                                 # the other word never saw it
    assert L.rk_attn_decode_noalloc_status() == 0
    got = call()
    assert (got.float() - want.float()).abs().max() < 2e-2


def test_a_failed_launch_is_reported_once():
    """A launch that the runtime refuses on the host (the default stream, while a stream that synchronizes with it is captured) returns
    its error, and the calls after it, which succeed, do not report it again."""
    rt = C.CDLL("libcudart.so.12")                                      # the one torch has loaded
    L = rk.lib()
    x = torch.randn(4, 64, device="cuda")
    codes, scales = torch.empty(4, 64, dtype=torch.uint8, device="cuda"), torch.empty(4, 2, dtype=torch.uint8, device="cuda")
    kt, kts = torch.zeros(64, 32, dtype=torch.uint8, device="cuda"), torch.zeros(2, 32, dtype=torch.uint8, device="cuda")
    k, ks = torch.empty(32, 64, dtype=torch.uint8, device="cuda"), torch.empty(32, 2, dtype=torch.uint8, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    stream, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 0) == 0
    try:
        refused = L.rk_mx_quantize(p(x), 4, 64, 0, p(codes), p(scales), None)
    finally:
        rt.cudaStreamEndCapture(stream, C.byref(graph))                 # the capture is invalid: an error, and no graph
        rt.cudaGetLastError()
        rt.cudaStreamDestroy(stream)
    assert refused > 0
    assert L.rk_import_kt_blocks(p(kt), p(kts), 1, 1, 32, 64, p(k), p(ks), None) == 0
    assert L.rk_mx_quantize(p(x), 4, 64, 0, p(codes), p(scales), None) == 0
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("form", [PAIRS, TURNS, SPLIT])
@pytest.mark.parametrize("shape", [(2, 4, 2, 1024, 128, False), (1, 2, 1, 640, 64, False), (1, 4, 4, 512, 128, True),      # no more query tiles than SMs
                                   (2, 16, 4, 900, 128, False), (1, 40, 8, 520, 64, False), (1, 52, 4, 384, 128, True)])  # more
def test_schedule_perturbation_leaves_every_bit_of_o(shape, form):
    """A few hundred nanoseconds of sleep at every key tile in one warp role at a time (softmax of query tile A,
    of tile B -- of the lower and of the upper keys, or of the even and the odd key tiles, where a CTA has one query tile --, correction, TMA producer,
    Q K^T issuer, P V issuer): if a hand-off between roles lacked a barrier the delayed
    role would read or overwrite something too early and O would change.  In every form, against the form the library chooses."""
    B, H, Hkv, S, d, cap = shape
    L = rk.lib()
    Q, K, V = randn_qkv(B, H, Hkv, S, S, d, seed=92)
    qc, qs, kc, ks, vc, vs = quantize_inputs(Q, K, V)
    kw = dict(causal=True, softcap=30.0 if cap else 0.0)
    base = rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
    try:
        with prefill_form(form):
            for role in (1, 2, 3, 4, 5, 6):
                L.rk_debug_set_prefill_perturb(role)
                for _ in range(2):
                    assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw), base), role
    finally:
        L.rk_debug_set_prefill_perturb(0)
    assert rk.last_device_status() == 0


# heads, queries, d, cap, options; heads 0: as many as it takes to have at least three items per SM
@pytest.mark.parametrize("shape", [(0, 100, 128, 0.0, {}), (0, 384, 64, 0.0, {}), (0, 200, 128, 30.0, dict(causal=False)), (0, 700, 128, 0.0, dict(window=150)),
                                   (0, 390, 128, 0.0, dict(q_pos0=-130)),
                                   (4, 600, 256, 0.0, {}), (0, 100, 256, 0.0, {}), (0, 128, 256, 50.0, dict(causal=False)), (0, 300, 256, 50.0, {}),
                                   (0, 640, 256, 0.0, dict(causal=False)), (0, 390, 256, 0.0, dict(q_pos0=-130)), (0, 700, 256, 0.0, dict(window=150))])
def test_schedule_perturbation_where_ctas_take_item_after_item(shape):
    """The same where a CTA goes on to other items, with a seventh role, O's way out (in it the delays lie between chunks, and before what the softmax
    warps leave behind of an item), and at d = 256: softmax group 0, group 1, the upper keys' warps of both, TMA producer, the issuers, O's way out.
    Items of one key tile and of none, odd and even numbers of them; O and the log-sum-exps."""
    H, S, d, cap, kw = shape
    L = rk.lib()
    if H == 0:
        per_head = (S + 127) // 128 if d == 256 else (S + 255) // 256
        H = -(-3 * torch.cuda.get_device_properties(0).multi_processor_count // per_head)
    qc, qs, kc, ks, vc, vs = quantize_inputs(*randn_qkv(1, H, H, S, S, d, seed=94))
    kw = dict(dict(causal=True, softcap=cap), **kw)
    lse0, lse = torch.empty(1, H, S, device="cuda"), torch.empty(1, H, S, device="cuda")
    base = rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=lse0, **kw)
    try:
        for role in (1, 2, 3, 4, 5, 6, 7):
            L.rk_debug_set_prefill_perturb(role)
            for _ in range(2):
                assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=lse, **kw), base), role
                assert torch.equal(lse, lse0), role
    finally:
        L.rk_debug_set_prefill_perturb(0)
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("shape", [(118, 300, 128, 0.0, {}), (88, 390, 64, 0.0, dict(q_pos0=-130)), (58, 700, 128, 0.0, dict(window=150)), (80, 500, 128, 30.0, {}),
                                   (420, 100, 64, 0.0, dict(causal=False)),           # one query tile at a time, key tiles in turn
                                   (240, 500, 128, 0.0, {}), (300, 300, 64, 30.0, {})])        # pairs
def test_schedule_perturbation_in_both_kernels_of_narrow_heads(shape):
    """The delays of the test above where a CTA has some three query tiles one after the other, and where it has as many pairs of them."""
    H, S, d, cap, kw = shape
    test_schedule_perturbation_where_ctas_take_item_after_item((H, S, d, cap, kw))


# heads, KV heads, queries, keys, d, V scaled along the keys, options
PREPARED = [(2, 2, 100, 128, 64, False, {}), (8, 2, 130, 100, 128, False, dict(causal=False)), (3, 3, 128, 128, 128, True, {}), (2, 1, 70, 90, 64, True, dict(causal=False)),
            (2, 2, 256, 256, 64, False, dict(causal=False)), (6, 2, 200, 250, 128, False, dict(q_pos0=50)), (4, 2, 256, 256, 128, True, {}), (2, 2, 129, 200, 64, True, dict(q_pos0=71)),
            (16, 16, 300, 384, 128, False, dict(causal=False)), (16, 16, 384, 300, 128, False, dict(window=150)), (4, 2, 300, 300, 64, False, dict(q_pos0=-130)),
            (6, 3, 384, 384, 64, False, {}), (4, 2, 260, 380, 128, True, dict(causal=False)), (4, 4, 300, 384, 64, True, dict(window=100, q_pos0=84))]


def _prepared(H, Hkv, Sq, Skv, d, along_keys, kw, fmt=rk.E4M3):
    """Operands, options and, asked of the library, that the attention kernel of this call prepares its operands itself."""
    axis = rk.V_SCALES_ALONG_KEYS if along_keys else rk.V_SCALES_ALONG_D
    kw = dict(dict(causal=True), **kw, v_scale_axis=axis, q_fmt=fmt, kv_fmt=fmt)
    a = PrefillArgs()
    a.B, a.H, a.H_kv, a.S_q, a.S_kv, a.d, a.v_scale_axis, a.q_fmt, a.kv_fmt = 1, H, Hkv, Sq, Skv, d, axis, fmt, fmt
    a.causal, a.q_pos0, a.window = int(kw["causal"]), kw.get("q_pos0", 0), kw.get("window", 0)
    assert rk.lib().rk_debug_prefill_prepares(C.byref(a))
    return quantize_inputs(*randn_qkv(1, H, Hkv, Sq, Skv, d, seed=98), axis, fmt), kw


@pytest.mark.parametrize("fmt", [rk.E4M3, rk.E5M2])
@pytest.mark.parametrize("shape", PREPARED)
def test_schedule_perturbation_where_the_kernel_prepares_its_operands(shape, fmt):
    """The same in calls of one to three key tiles, with two roles more: the warps that put the scales of Q and K into atoms and those that re-block V, or put its scales into atoms."""
    (qc, qs, kc, ks, vc, vs), kw = _prepared(*shape, fmt=fmt)
    H, S = shape[0], shape[2]
    lse0, lse = torch.empty(1, H, S, device="cuda"), torch.empty(1, H, S, device="cuda")
    base = rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=lse0, **kw)
    try:
        for role in (1, 2, 3, 4, 5, 6, 7, 8, 9):
            rk.lib().rk_debug_set_prefill_perturb(role)
            for _ in range(2):
                assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, lse=lse, **kw), base), role
                assert torch.equal(lse, lse0), role
    finally:
        rk.lib().rk_debug_set_prefill_perturb(0)
    assert rk.last_device_status() == 0


@pytest.mark.parametrize("shape", [PREPARED[0], PREPARED[3], PREPARED[5], PREPARED[6], PREPARED[8], PREPARED[12]])
def test_a_preparation_that_is_not_handed_over_ends_the_call_and_the_next_one_is_whole(shape):
    """Some of the warps that prepare the operands do not hand over (scale atoms of K; keys of V's tiles, the scales of its last tile): the waits for them run out, with the
    other roles' behind them, the call ends and the next one has every bit."""
    (qc, qs, kc, ks, vc, vs), kw = _prepared(*shape)
    L = rk.lib()
    want = rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
    assert rk.last_device_status() == 0
    for role in (8, 9):
        L.rk_debug_set_prefill_perturb(100 + role)
        try:
            rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
            torch.cuda.synchronize()
        finally:
            L.rk_debug_set_prefill_perturb(0)
            status = rk.last_device_status()
        assert 100 < status < 600, (role, status)
        assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw), want), role
        assert rk.last_device_status() == 0


@pytest.mark.parametrize("shape", [PREPARED[4], PREPARED[6], PREPARED[8], PREPARED[12]])
def test_a_role_that_gives_up_where_the_kernel_prepares_its_operands(shape):
    """The roles of the other tests, in calls of two and three key tiles of this kind: without a mask, so that all have a second tile."""
    (qc, qs, kc, ks, vc, vs), kw = _prepared(*shape[:-1], dict(causal=False))
    L = rk.lib()
    want = rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
    assert rk.last_device_status() == 0
    for role in (1, 2, 3, 4, 5, 6):
        L.rk_debug_set_prefill_perturb(100 + role)
        try:
            rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw)
            torch.cuda.synchronize()
        finally:
            L.rk_debug_set_prefill_perturb(0)
            status = rk.last_device_status()
        assert 100 < status < 600, (role, status)
        assert torch.equal(rk.attn_prefill(qc, kc, vc, qs, ks, vs, **kw), want), role
        assert rk.last_device_status() == 0


def test_tensor_pipe_ceiling_loop_never_runs_into_its_waits():
    """The GEMM-only loop bench.py measures the tensor-pipe ceiling with paces itself through two alternating
    mbarriers (one barrier per batch in flight: a barrier that completes two phases before its waiter looks reads as
    "not yet", and a single pacing barrier did that about once in 10 000 launches).  A few thousand launches, short
    and long, must leave the device status word at zero."""
    import ctypes as C
    L = rk.lib()
    if not hasattr(L, "rk_debug_mxfp8_mma_loop"):
        pytest.skip("measurement aid not exported")
    L.rk_debug_mxfp8_mma_loop.restype = C.c_int
    L.rk_debug_mxfp8_mma_loop.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    tiles = torch.randint(0, 0x7E, (2, 128 * 128), dtype=torch.uint8, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for iters, n in ((64, 500), (200, 1500), (1024, 500), (8192, 100)):
        for _ in range(n):
            assert L.rk_debug_mxfp8_mma_loop(C.c_void_p(tiles[0].data_ptr()), C.c_void_p(tiles[1].data_ptr()), iters, st) == 0
        torch.cuda.synchronize()
        assert rk.last_device_status() == 0, iters
