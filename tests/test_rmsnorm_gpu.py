"""RMSNorm fused with the MX quantizer (the QKV-projection prologue of kernels/rmsnorm_qkv_fused) on the GPU: codes and
scales bit-exact with the reference's rmsnorm golden followed by the block quantizer."""
import contextlib
import os

import numpy as np
import pytest
import torch

import oracle
import radiance_kernels_b200 as rk
from helpers import np_

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def _expect(x, gamma, eps, fmt, unit):
    y = oracle.rmsnorm(x, gamma, eps)
    if unit:
        L = oracle.lib()
        codes = np.array([L.rko_encode_elem_rne(float(v), fmt) for v in y.ravel()], np.uint8).reshape(y.shape)
        return codes, np.full((y.shape[0], y.shape[1] // 32), 0x7F, np.uint8)
    return oracle.quantize(y, fmt)


def test_reference_golden_inputs_bit_exact():
    """The inputs of the committed rmsnorm fixture (made by importing lib/golden/golden.py): normalized values that
    equal the reference's bit for bit go through the same block rule, so codes and scales must match exactly."""
    z = np.load(os.path.join(GOLDEN, "rmsnorm_vectors.npz"))
    for i in range(4):
        x, g, eps = z[f"x{i}"], z[f"g{i}"], float(z[f"eps{i}"])
        if x.shape[1] % 32:
            continue
        want_c, want_s = oracle.quantize(z[f"y{i}"])
        c, s = rk.rmsnorm_mx_quantize(torch.from_numpy(x).cuda(), torch.from_numpy(g).cuda(), eps)
        assert np.array_equal(np_(c), want_c) and np.array_equal(np_(s), want_s), i


@pytest.mark.parametrize("rows,K,fmt,unit,bf16", [(64, 256, 0, True, True), (100, 4096, 0, False, False), (33, 128, 3, False, False),
                                                  (257, 1024, 1, False, True), (1, 32, 0, False, False), (70, 2048, 2, False, False),
                                                  (48, 512, 4, False, False), (96, 256, 4, False, True)])
def test_rmsnorm_quantize_matches_oracle(rows, K, fmt, unit, bf16):
    rng = np.random.default_rng(rows * 7 + K)
    x = (rng.standard_normal((rows, K)) * np.exp2(rng.integers(-6, 7, (rows, 1)))).astype(np.float32)
    gamma = (0.75 + 0.5 * rng.random(K)).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    if bf16:
        xt = xt.bfloat16()
        x = np_(xt.float())
    eps = 1e-5
    want_c, want_s = _expect(x, gamma, eps, fmt, unit)
    c, s = rk.rmsnorm_mx_quantize(xt, torch.from_numpy(gamma).cuda(), eps, fmt=fmt, unit_scale=unit)
    torch.cuda.synchronize()
    assert np.array_equal(np_(s), want_s)
    assert np.array_equal(np_(c), want_c)


def test_zero_rows_and_huge_rows():
    """An all-zero row normalizes to zeros (rms = 1/sqrt(eps)); a row of large values stays finite."""
    x = np.zeros((3, 64), np.float32)
    x[1] = 3.0e18
    x[2, 5] = -1.0e-30
    gamma = np.ones(64, np.float32)
    want_c, want_s = oracle.quantize(oracle.rmsnorm(x, gamma, 1e-6))
    c, s = rk.rmsnorm_mx_quantize(torch.from_numpy(x).cuda(), torch.from_numpy(gamma).cuda(), 1e-6)
    assert np.array_equal(np_(c), want_c) and np.array_equal(np_(s), want_s)


@pytest.mark.parametrize("rows,K,bf16,shift,inf_gamma", [(1, 96, True, 0, False), (593, 288, False, 0, True), (593, 544, True, 2, False),
                                                         (9473, 64, True, 0, True), (2400, 800, False, 1, False), (3, 66592, True, 0, False)])
def test_row_groups_chunks_and_alignment(rows, K, bf16, shift, inf_gamma):
    """Ragged row groups (one CTA slot per row and one row more, two waves), ragged column chunks, a base that is only 4-byte
    aligned, scale rows too long to meet in shared memory, and an infinite gamma (blocks that need the integer encoder)."""
    rng = np.random.default_rng(rows + K)
    x = rng.standard_normal((rows, K)).astype(np.float32)
    gamma = (0.75 + 0.5 * rng.random(K)).astype(np.float32)
    if inf_gamma:
        gamma[K // 2] = np.inf
    flat = torch.empty(rows * K + shift, dtype=torch.bfloat16 if bf16 else torch.float32, device="cuda")
    xt = flat[shift:].view(rows, K)
    xt.copy_(torch.from_numpy(x))
    want_c, want_s = _expect(np_(xt.float()), gamma, 1e-5, 0, False)
    c, s = rk.rmsnorm_mx_quantize(xt, torch.from_numpy(gamma).cuda(), 1e-5)
    assert np.array_equal(np_(s), want_s)
    assert np.array_equal(np_(c), want_c)


@pytest.mark.parametrize("rows,K,fmt,unit", [(1, 2048, 0, False), (33, 2080, 0, False), (9473, 2048, 0, False), (4099, 1024, 0, True), (298, 4128, 3, False)])
def test_bf16_rows_by_bulk_copy(rows, K, fmt, unit):
    """One row and one wave of row groups and more, rows that end inside a piece of 1024 bytes, more pieces than the ring holds; rows of zeros, of values whose
    squares are subnormal or overflow, and blocks with a NaN or an infinity."""
    rng = np.random.default_rng(rows + K)
    x = (rng.standard_normal((rows, K)) * np.exp2(rng.integers(-6, 7, (rows, 1)))).astype(np.float32)
    if rows > 10:
        x[3] = 0.0
        x[5] *= 2.0 ** -70
        x[7, ::3] *= 2.0 ** 62
        x[9, K - 40] = np.inf
        x[10, 17] = np.nan
    gamma = (0.75 + 0.5 * rng.random(K)).astype(np.float32)
    xt = torch.from_numpy(x).cuda().bfloat16()
    want_c, want_s = _expect(np_(xt.float()), gamma, 1e-5, fmt, unit)
    c, s = rk.rmsnorm_mx_quantize(xt, torch.from_numpy(gamma).cuda(), 1e-5, fmt=fmt, unit_scale=unit)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    assert np.array_equal(np_(s), want_s)
    got_c = np_(c).copy()
    if rows > 10:                                      # rows 9 and 10: inf x 0 and sums with a NaN; x86 and the GPU give such a NaN different signs, the codes keep them
        sign = 0x80 if fmt == 0 else 0x20
        got_c[9:11] &= ~np.uint8(sign)
        want_c[9:11] &= ~np.uint8(sign)
    assert np.array_equal(got_c, want_c)


@pytest.mark.parametrize("rows,K,bf16,fmt,unit", [(1, 1056, True, 0, False), (1, 4096, False, 0, True), (37, 4128, True, 0, False), (445, 2080, False, 1, False), (889, 1536, True, 0, False),
                                                  (1777, 1792, True, 2, False), (3552, 1056, True, 0, False), (900, 8224, True, 4, False), (30, 12288, False, 3, False),
                                                  (12, 50016, True, 0, False), (12, 50016, False, 0, False)])
def test_chains_cut_into_segments(rows, K, bf16, fmt, unit):
    """Rows whose index-order sums are taken by segments: one to eight of them to a CTA, segments of a warp and of several, ragged last segments.  Sums that
    stay in a binade for long, cross several in one segment, start late, tie at nearly every addition, cannot be guessed (the share of one value), overflow or hold a NaN."""
    rng = np.random.default_rng(rows + K)
    x = (rng.standard_normal((rows, K)) * np.exp2(rng.integers(-6, 7, (rows, 1)))).astype(np.float32)
    ramp = np.exp2(np.linspace(-40, 40, K)).astype(np.float32)
    forms = [lambda v: 0 * v, lambda v: v * 2.0 ** -70, lambda v: v * 2.0 ** -45, lambda v: v * ramp, lambda v: v * ramp[::-1], lambda v: np.sign(v), lambda v: np.sign(v) * 1.5,
             lambda v: np.where(np.arange(K) < K // 2, 0, v), lambda v: np.where(np.arange(K) % 97, v * 2.0 ** -30, v), lambda v: np.where(np.arange(K) == K // 3, 3.0e4, v),
             lambda v: np.where(np.arange(K) % 3, v, v * 2.0 ** 62), lambda v: np.round(v * 4) / 4]
    for i, f in enumerate(forms):
        if i < rows:
            x[i * (rows // min(rows, len(forms)))] = f(x[i * (rows // min(rows, len(forms)))])
    if rows > 30:
        x[rows - 2, K - 40] = np.inf
        x[rows - 1, 17] = np.nan
    gamma = (0.75 + 0.5 * rng.random(K)).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    xt = xt.bfloat16() if bf16 else xt
    want_c, want_s = _expect(np_(xt.float()), gamma, 1e-5, fmt, unit)
    c, s = rk.rmsnorm_mx_quantize(xt, torch.from_numpy(gamma).cuda(), 1e-5, fmt=fmt, unit_scale=unit)
    torch.cuda.synchronize()
    assert rk.last_device_status() == 0
    got_c = np_(c).copy()
    if rows > 30:                                      # signs of NaN: as in the test above
        sign = (0x80, 0x80, 0x20, 0x20, 0x08)[fmt]
        got_c[-2:] &= ~np.uint8(sign)
        want_c[-2:] &= ~np.uint8(sign)
    assert np.array_equal(np_(s), want_s)
    assert np.array_equal(got_c, want_c)


@pytest.mark.parametrize("rows,K,first", [(4500, 2048, 1.0), (4500, 2048, 0.0), (4500, 4096, 2.0 ** -50), (4500, 2080, 2.0 ** -51)])
def test_fused_chains_of_large_calls(rows, K, first):
    """Rows that begin with an element from which on a fused multiply-add gives the bits of a product and a sum, and rows that do not: beside elements whose
    squares round to subnormal numbers, and sums that stay small."""
    rng = np.random.default_rng(rows + K)
    x = rng.standard_normal((rows, K)).astype(np.float32)
    x[::3] *= np.exp2(rng.integers(-75, -45, (rows, K)))[::3]
    x[:, 0] = first
    gamma = (0.75 + 0.5 * rng.random(K)).astype(np.float32)
    xt = torch.from_numpy(x).cuda().bfloat16()
    want_c, want_s = _expect(np_(xt.float()), gamma, 1e-30, 0, False)
    c, s = rk.rmsnorm_mx_quantize(xt, torch.from_numpy(gamma).cuda(), 1e-30)
    torch.cuda.synchronize()
    assert np.array_equal(np_(s), want_s)
    assert np.array_equal(np_(c), want_c)


STAGED, RING, SEGMENTS = 1, 2, 3


@contextlib.contextmanager
def rmsnorm_form(form):
    """RMSNorm calls take this form (rows staged through registers; by bulk copies in a ring, bf16 alone)."""
    rk.lib().rk_debug_set_rmsnorm_form(form)
    try:
        yield
    finally:
        rk.lib().rk_debug_set_rmsnorm_form(0)


@pytest.mark.parametrize("form,rows,K,bf16,fmt,unit", [
    (RING, 1, 2048, True, 0, False), (RING, 33, 2080, True, 0, False), (RING, 300, 1056, True, 1, False), (RING, 37, 4128, True, 2, True), (RING, 298, 4128, True, 3, False),
    (RING, 64, 12288, True, 4, False), (RING, 597, 2048, True, 0, True),
    (STAGED, 100, 4096, False, 0, False), (STAGED, 445, 2080, False, 1, True), (STAGED, 70, 2048, False, 2, False), (STAGED, 37, 4128, False, 3, False),
    (STAGED, 300, 1056, False, 4, False), (STAGED, 593, 1536, False, 0, True),
    (STAGED, 3, 66592, True, 0, False), (STAGED, 297, 1536, True, 1, False), (STAGED, 64, 2048, True, 4, True)])
def test_the_forms_of_large_calls_on_rows_that_segments_take(form, rows, K, bf16, fmt, unit):
    """The kernels that calls of more rows take, in every format, on the rows of the test of the segments: such calls are too large to check in number.  Ragged row groups and pieces, more
    pieces than the ring holds, scale rows too long to meet in shared memory."""
    assert rk.lib().rk_debug_rmsnorm_form(rows, K, bf16, 0) == SEGMENTS
    with rmsnorm_form(form):
        assert rk.lib().rk_debug_rmsnorm_form(rows, K, bf16, 0) == form
        test_chains_cut_into_segments(rows, K, bf16, fmt, unit)


@pytest.mark.parametrize("form,rows,K,bf16,fmt,unit", [(STAGED, 3600, 1056, False, 0, False), (RING, 9473, 2048, True, 1, False), (STAGED, 300, 1024, False, 2, False)])
def test_the_forms_that_calls_take_by_themselves(form, rows, K, bf16, fmt, unit):
    """fp32 rows of more than 1024 columns, more of them than lie on the chip at once; bf16 rows of a whole wave; short rows."""
    if torch.cuda.get_device_properties(0).multi_processor_count <= 160:
        assert rk.lib().rk_debug_rmsnorm_form(rows, K, bf16, 0) == form
    test_chains_cut_into_segments(rows, K, bf16, fmt, unit)


def _us_per_call(call, calls=20):
    """Median of replays of a graph of calls: neither the host nor a neighbour on the machine counts."""
    call()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(calls):
            call()
    times = []
    for _ in range(15):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        graph.replay()
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end) * 1000 / calls)
    return sorted(times)[len(times) // 2]


@pytest.mark.parametrize("rows,K,bf16", [(1, 4096, True), (300, 12288, True), (1, 4096, False), (300, 4096, False)])
@pytest.mark.parametrize("kind", ["tiny", "nan", "inf"])
def test_rows_that_are_added_as_they_lie_cost_a_chain(rows, K, bf16, kind):
    """Rows whose sums stay below 2^-87 or hold a NaN or an infinity have no binade to take segments in, and one lane adds them up in the end: at the pace of the kernel that walks
    every chain as it lies, plus the two passes over the segments (1.0-1.2 of its time; 2-4 where a segment at a time was looked up and added)."""
    g = torch.Generator(device="cuda").manual_seed(97)
    x = torch.randn(rows, K, generator=g, device="cuda")
    if kind == "tiny":
        x *= 2.0 ** -52
    else:
        x[:, 17] = float(kind)
    x = x.bfloat16() if bf16 else x
    gamma = torch.rand(K, generator=g, device="cuda") + 0.5
    assert rk.lib().rk_debug_rmsnorm_form(rows, K, bf16, 0) == SEGMENTS
    segments = _us_per_call(lambda: rk.rmsnorm_mx_quantize(x, gamma, 1e-5))
    with rmsnorm_form(RING if bf16 else STAGED):
        chain = _us_per_call(lambda: rk.rmsnorm_mx_quantize(x, gamma, 1e-5))
    assert segments < 1.7 * chain, (segments, chain)
