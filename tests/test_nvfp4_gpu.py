"""Parity of the NVFP4 tcgen05 GEMM (through the C ABI) with the CPU oracle.

Tolerance (from the task statement): dequantised values bit-exact; bf16 outputs
within max relative error 2e-2 per element.  Products of e2m1 codes and e4m3
scales are exact and the tensor core accumulates in fp32, so in practice the
only difference from the oracle is the final bf16 rounding: the test also
requires agreement within one bf16 ulp of the binary64-accumulated value.
"""
import ctypes as C
import os

import numpy as np
import pytest

from makepad_b200 import _lib, synth

pytestmark = pytest.mark.gpu
TOL = 2e-2
GOLD = os.path.join(os.path.dirname(__file__), "golden", "nvfp4_small.npz")


def _gemm(ctx, a, sfa, ta, b, sfb, tb):
    import torch
    import makepad_b200
    w = makepad_b200.Nvfp4Weight(ctx, b, sfb, tb)
    y = makepad_b200.QuantLinear(w)((torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda(), ta))
    torch.cuda.synchronize()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
    out = y.view(torch.int16).cpu().numpy().view(np.uint16)
    w.destroy()
    return out


def _check(orc, got_bits, c32):
    got = orc.bf16_bits_to_f32(got_bits).astype(np.float64)
    ref = c32.astype(np.float64)
    strict, floored = orc.rel_err(got, ref)
    assert floored < TOL, (strict, floored)
    # within one bf16 ulp of the exact value (2^-8 relative), plus fp32 accumulation noise
    rms = np.sqrt(np.mean(ref * ref)) + 1e-30
    assert np.all(np.abs(got - ref) <= np.abs(ref) * 2.0 ** -8 + 1e-5 * rms)


@pytest.mark.parametrize("R,K", [(1, 16), (5, 48), (224, 256), (300, 4096)])
def test_dequant_bit_exact(ctx, orc, R, K):
    import torch
    codes, sf = synth.nvfp4_tensor(R, K, seed=R + K)
    out = torch.empty((R, K), dtype=torch.float32, device="cuda")
    cd, sd = torch.from_numpy(codes).cuda(), torch.from_numpy(sf).cuda()
    for ts in (1.0, 0.37):
        ctx.check(ctx.lib.mpq_nvfp4_dequantize(ctx.h, R, K, cd.data_ptr(), sd.data_ptr(), C.c_float(ts), out.data_ptr(), None))
        torch.cuda.synchronize()
        want = orc.nvfp4_dequantize(codes, sf, ts)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_dequant_every_code_and_scale(ctx, orc):
    import torch
    # 16 codes x all 127 finite non-negative scales (and the negative ones too)
    sfb = np.arange(256, dtype=np.uint8)
    sfb = sfb[(sfb & 0x7F) != 0x7F]
    codes = synth.pack_nibbles(np.tile(np.arange(16, dtype=np.uint8), (len(sfb), 1)))
    sf = sfb[:, None].copy()
    out = torch.empty((len(sfb), 16), dtype=torch.float32, device="cuda")
    cd, sd = torch.from_numpy(codes).cuda(), torch.from_numpy(sf).cuda()
    ctx.check(ctx.lib.mpq_nvfp4_dequantize(ctx.h, len(sfb), 16, cd.data_ptr(), sd.data_ptr(), C.c_float(1.0), out.data_ptr(), None))
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), orc.nvfp4_dequantize(codes, sf, 1.0).view(np.uint32))


def test_weight_export_bit_exact(ctx, orc):
    import makepad_b200
    b, sfb = synth.nvfp4_tensor(448, 512, seed=3)
    w = makepad_b200.Nvfp4Weight(ctx, b, sfb, 0.25)
    assert np.array_equal(w.dequantize().cpu().numpy().view(np.uint32), orc.nvfp4_dequantize(b, sfb, 0.25).view(np.uint32))


@pytest.mark.parametrize("M,N,K", [(128, 224, 256), (128, 224, 1024), (256, 448, 512), (384, 672, 2048),
                                   (100, 200, 320), (1, 8, 32), (129, 232, 288), (2048, 224, 4096)])
def test_gemm_matches_oracle(ctx, orc, M, N, K):
    a, sfa = synth.nvfp4_tensor(M, K, seed=M, stream=0)
    b, sfb = synth.nvfp4_tensor(N, K, seed=M, stream=1)
    c32, c16 = orc.nvfp4_gemm(a, sfa, 0.5, b, sfb, 3.0)
    got = _gemm(ctx, a, sfa, 0.5, b, sfb, 3.0)
    _check(orc, got, c32)
    # the rounding itself agrees with the oracle's on nearly every element (ties in fp32 accumulation order aside)
    assert np.mean(got == c16) > 0.99


@pytest.mark.parametrize("kernel", ["single", "pair"])
@pytest.mark.parametrize("M,N,K", [(128, 224, 256), (256, 448, 512), (100, 200, 320), (1, 8, 32), (640, 672, 2048),
                                   (300, 224, 4096), (1200, 2912, 1024), (16, 448, 4096), (64, 232, 288)])
def test_single_cta_kernel_matches_oracle(ctx, orc, kernel, M, N, K):
    """The one-CTA-per-tile kernel, used where clusters of two cannot be scheduled (MPQ_FP4_KERNEL=single), and the one of CTA pairs, which
    calls of up to 64 rows take where the weight has no tensor maps (pair), compute the same GEMM."""
    a, sfa = synth.nvfp4_tensor(M, K, seed=M + 2, stream=0)
    b, sfb = synth.nvfp4_tensor(N, K, seed=M + 2, stream=1)
    c32, c16 = orc.nvfp4_gemm(a, sfa, 0.5, b, sfb, 3.0)
    os.environ["MPQ_FP4_KERNEL"] = kernel
    try:
        got = _gemm(ctx, a, sfa, 0.5, b, sfb, 3.0)
    finally:
        del os.environ["MPQ_FP4_KERNEL"]
    _check(orc, got, c32)
    assert np.mean(got == c16) > 0.99


def test_many_tiles_per_cta_deterministic(ctx, orc):
    """More tiles than CTA pairs (every pair runs several tiles back to back) and K % 256 != 0 (re-tiled activation scales):
    equal to the oracle and bit-identical between runs and between the two kernels."""
    M, N, K = 1536, 224 * 40, 1056
    a, sfa = synth.nvfp4_tensor(M, K, seed=11, stream=0)
    b, sfb = synth.nvfp4_tensor(N, K, seed=11, stream=1)
    c32, _ = orc.nvfp4_gemm(a, sfa, 1.0, b, sfb, 1.0)
    got = _gemm(ctx, a, sfa, 1.0, b, sfb, 1.0)
    _check(orc, got, c32)
    for _ in range(3):
        assert np.array_equal(_gemm(ctx, a, sfa, 1.0, b, sfb, 1.0), got)
    os.environ["MPQ_FP4_KERNEL"] = "single"
    try:
        assert np.array_equal(_gemm(ctx, a, sfa, 1.0, b, sfb, 1.0), got)
    finally:
        del os.environ["MPQ_FP4_KERNEL"]


def test_known_answers(ctx, orc):
    M, N, K = 128, 224, 256
    one = lambda R: synth.pack_nibbles(np.full((R, K), 2, dtype=np.uint8))
    sf1 = lambda R: np.full((R, K // 16), 0x38, dtype=np.uint8)
    got = orc.bf16_bits_to_f32(_gemm(ctx, one(M), sf1(M), 1.0, one(N), sf1(N), 1.0))
    assert np.all(got == float(K))
    # zero scales zero their blocks; +-0 codes contribute nothing
    z = np.zeros((M, K // 16), dtype=np.uint8)
    assert np.all(orc.bf16_bits_to_f32(_gemm(ctx, one(M), z, 1.0, one(N), sf1(N), 1.0)) == 0.0)
    negzero = synth.pack_nibbles(np.full((M, K), 8, dtype=np.uint8))
    assert np.all(orc.bf16_bits_to_f32(_gemm(ctx, negzero, sf1(M), 1.0, one(N), sf1(N), 1.0)) == 0.0)
    # max magnitudes: 6 * 448 on both sides, K = 256 terms: 256 * (6*448)^2 = 1.85e9 fits fp32 and bf16
    six = lambda R: synth.pack_nibbles(np.full((R, K), 7, dtype=np.uint8))
    big = lambda R: np.full((R, K // 16), 0x7E, dtype=np.uint8)
    got = orc.bf16_bits_to_f32(_gemm(ctx, six(M), big(M), 1.0, six(N), big(N), 1.0))
    want = orc.bf16_bits_to_f32(orc.f32_to_bf16(np.array([256.0 * (6 * 448.0) ** 2], dtype=np.float32)))[0]
    assert np.all(got == want)


def test_golden_vectors(ctx, orc):
    g = np.load(GOLD)
    n = len([k for k in g.files if k.endswith("_sfa")])
    for i in range(n):
        got = _gemm(ctx, g[f"fp4_{i}_a"], g[f"fp4_{i}_sfa"], 1.0, g[f"fp4_{i}_b"], g[f"fp4_{i}_sfb"], 1.0)
        _check(orc, got, g[f"fp4_{i}_c32"])


def test_prefill_shape_rows_against_oracle(ctx, orc):
    """Configuration 3 at full size (2048 x 4096 x 14336); the oracle checks a sample of 48 rows of A."""
    import torch
    import makepad_b200
    M, N, K = 2048, 14336, 4096
    a, sfa = synth.nvfp4_tensor(M, K, seed=0, stream=0)
    b, sfb = synth.nvfp4_tensor(N, K, seed=0, stream=1)
    w = makepad_b200.Nvfp4Weight(ctx, b, sfb, 1.0)
    lin = makepad_b200.QuantLinear(w)
    ad, sd = torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda()
    y = lin((ad, sd, 1.0))
    y2 = lin((ad, sd, 1.0))
    torch.cuda.synchronize()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
    assert torch.equal(y, y2)                                         # deterministic
    rows = np.random.default_rng(0).choice(M, 48, replace=False)
    c32, _ = orc.nvfp4_gemm(a[rows], sfa[rows], 1.0, b, sfb, 1.0)
    got = y[torch.from_numpy(rows).cuda()].view(torch.int16).cpu().numpy().view(np.uint16)
    _check(orc, got, c32)
    # size-independent property at full size: scaling A's tensor scale by 2 doubles every output exactly
    y3 = lin((ad, sd, 2.0))
    torch.cuda.synchronize()
    assert torch.equal(y3.float(), 2.0 * y.float())


def test_error_statuses(ctx):
    import torch
    lib = ctx.lib
    b, sfb = synth.nvfp4_tensor(224, 256, seed=1)
    h = C.c_void_p()
    assert lib.mpq_nvfp4_weight_create(ctx.h, 224, 240, b.ctypes.data, sfb.ctypes.data, C.c_float(1.0), C.byref(h)) == _lib.ERR_SHAPE
    assert lib.mpq_nvfp4_weight_create(ctx.h, 220, 256, b.ctypes.data, sfb.ctypes.data, C.c_float(1.0), C.byref(h)) == _lib.ERR_SHAPE
    assert lib.mpq_nvfp4_weight_create(ctx.h, 224, 256, None, sfb.ctypes.data, C.c_float(1.0), C.byref(h)) == _lib.ERR_INVALID_ARG
    assert lib.mpq_nvfp4_weight_create(ctx.h, 224, 256, b.ctypes.data, sfb.ctypes.data, C.c_float(1.0), C.byref(h)) == _lib.OK
    a = torch.zeros(128 * 128 + 16, dtype=torch.uint8, device="cuda")
    c = torch.zeros(128 * 224, dtype=torch.bfloat16, device="cuda")
    assert lib.mpq_nvfp4_gemm_forward(ctx.h, h, a.data_ptr() + 1, a.data_ptr(), C.c_float(1.0), 128, c.data_ptr(), None) == _lib.ERR_ALIGN
    assert lib.mpq_nvfp4_gemm_forward(ctx.h, h, a.data_ptr(), a.data_ptr(), C.c_float(1.0), 0, c.data_ptr(), None) == _lib.ERR_SHAPE
    assert lib.mpq_nvfp4_gemm_forward(ctx.h, h, None, a.data_ptr(), C.c_float(1.0), 128, c.data_ptr(), None) == _lib.ERR_INVALID_ARG
    # a Q4 entry point refuses an NVFP4 weight
    x = torch.zeros(256, device="cuda")
    assert lib.mpq_q4_linear_forward(ctx.h, h, x.data_ptr(), 1, x.data_ptr(), None) == _lib.ERR_INVALID_ARG
    assert lib.mpq_weight_destroy(h) == _lib.OK


def test_output_guard_regions_untouched(ctx):
    """TMA tile stores clip at the tensor's edge: nothing is written outside C, for M and N off the tile grid."""
    import torch
    import makepad_b200
    M, N, K = 130, 232, 288
    a, sfa = synth.nvfp4_tensor(M, K, seed=21, stream=0)
    b, sfb = synth.nvfp4_tensor(N, K, seed=21, stream=1)
    w = makepad_b200.Nvfp4Weight(ctx, b, sfb, 1.0)
    buf = torch.full((M * N + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    c = buf[2048:2048 + M * N].view(M, N)
    for kernel in (None, "single"):
        buf.fill_(7.0)
        if kernel:
            os.environ["MPQ_FP4_KERNEL"] = kernel
        try:
            makepad_b200.QuantLinear(w)((torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda(), 1.0), out=c)
            torch.cuda.synchronize()
        finally:
            os.environ.pop("MPQ_FP4_KERNEL", None)
        assert (buf[:2048] == 7.0).all() and (buf[2048 + M * N:] == 7.0).all()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
    w.destroy()


def test_error_metrics_strict_and_floored(ctx, orc):
    """Strict and floored (1e-2 and 1e-3 of the rms) maxima of the bf16 output against the exact value: all three are
    bounded by the bf16 rounding (2^-8), because the products are exact and the accumulation is fp32."""
    a, sfa = synth.nvfp4_tensor(256, 1024, seed=5, stream=0)
    b, sfb = synth.nvfp4_tensor(448, 1024, seed=5, stream=1)
    c32, _ = orc.nvfp4_gemm(a, sfa, 1.0, b, sfb, 1.0)
    got = orc.bf16_bits_to_f32(_gemm(ctx, a, sfa, 1.0, b, sfb, 1.0)).astype(np.float64)
    rep = orc.err_report(got, c32.astype(np.float64))
    print(f"NVFP4 256x448x1024: {rep}")
    assert rep["floored_1e-2_rms"] < TOL and rep["floored_1e-3_rms"] < TOL


def test_weight_export_reads_the_tiled_scales(ctx, orc):
    """The weight keeps its scale factors only in the tiled order the GEMM consumes; the export un-tiles them, so a
    bit-exact export proves the tiling pass (rows and K off the tile grid included)."""
    import makepad_b200
    for (N, K) in [(448, 512), (232, 288), (1000, 4096), (8, 32)]:
        b, sfb = synth.nvfp4_tensor(N, K, seed=N + K)
        w = makepad_b200.Nvfp4Weight(ctx, b, sfb, 0.5)
        assert np.array_equal(w.dequantize().cpu().numpy().view(np.uint32), orc.nvfp4_dequantize(b, sfb, 0.5).view(np.uint32))
        w.destroy()


@pytest.mark.parametrize("M,K", [(1, 16), (7, 48), (200, 512), (2048, 4096)])
def test_activation_quantisation_bit_exact(ctx, orc, M, K):
    """fp32 and bf16 activations -> NVFP4 on the GPU: the same bytes as the CPU checker, and usable as the GEMM's A."""
    import torch
    rng = np.random.default_rng(M + K)
    x = (rng.standard_normal((M, K)) * rng.uniform(1e-3, 50, size=(M, 1))).astype(np.float32)
    x[0, :16] = 0                                                    # an all-zero block
    if M > 1:
        x[1, :4] = [448 * 6 * 2, -1e-9, 0.25, 0.75]                  # saturation, underflow, ties
    for ts in (1.0, 0.37):
        for bf16 in (0, 1):
            xd = torch.from_numpy(x).cuda()
            if bf16:
                xd = xd.to(torch.bfloat16)
                want_c, want_s = orc.nvfp4_quantize(xd.float().cpu().numpy(), ts)
            else:
                want_c, want_s = orc.nvfp4_quantize(x, ts)
            codes = torch.empty((M, K // 2), dtype=torch.uint8, device="cuda")
            sf = torch.empty((M, K // 16), dtype=torch.uint8, device="cuda")
            ctx.check(ctx.lib.mpq_nvfp4_quantize_activations(ctx.h, C.c_void_p(xd.data_ptr()), bf16, M, K, C.c_float(ts),
                                                             C.c_void_p(codes.data_ptr()), C.c_void_p(sf.data_ptr()), None))
            torch.cuda.synchronize()
            assert np.array_equal(sf.cpu().numpy(), want_s)
            assert np.array_equal(codes.cpu().numpy(), want_c)
    assert ctx.lib.mpq_nvfp4_quantize_activations(ctx.h, C.c_void_p(xd.data_ptr()), 0, M, 24, C.c_float(1.0), C.c_void_p(codes.data_ptr()),
                                                  C.c_void_p(sf.data_ptr()), None) == _lib.ERR_SHAPE


def test_quantise_then_gemm(ctx, orc):
    """The prefill chain: quantise fp32 activations on the GPU, feed them to the GEMM; equal to the checker's chain."""
    import torch
    import makepad_b200
    M, N, K = 256, 448, 1024
    x = synth.activations(M, K, seed=17)
    b, sfb = synth.nvfp4_tensor(N, K, seed=17, stream=1)
    xd = torch.from_numpy(x).cuda()
    codes = torch.empty((M, K // 2), dtype=torch.uint8, device="cuda")
    sf = torch.empty((M, K // 16), dtype=torch.uint8, device="cuda")
    ctx.check(ctx.lib.mpq_nvfp4_quantize_activations(ctx.h, C.c_void_p(xd.data_ptr()), 0, M, K, C.c_float(1.0), C.c_void_p(codes.data_ptr()),
                                                     C.c_void_p(sf.data_ptr()), None))
    w = makepad_b200.Nvfp4Weight(ctx, b, sfb, 1.0)
    y = makepad_b200.QuantLinear(w)((codes, sf, 1.0))
    torch.cuda.synchronize()
    a_c, a_s = orc.nvfp4_quantize(x, 1.0)
    c32, _ = orc.nvfp4_gemm(a_c, a_s, 1.0, b, sfb, 1.0)
    _check(orc, y.view(torch.int16).cpu().numpy().view(np.uint16), c32)
    w.destroy()


@pytest.mark.parametrize("ts", [1.0, 0.37, 2.0 ** -64, 2.0 ** 64, 1e-25, 3e20])
def test_quantisation_at_the_rounding_boundaries(ctx, orc, ts):
    """Quotients on and a few ulp beside every boundary of the e2m1 grid, for every positive e4m3 scale, on the path with one
    reciprocal per block (tensor scale within 2^+-64) and on the path with divisions; then infinities and NaN."""
    import torch
    import makepad_b200
    ts = np.float32(ts)
    rows = []
    for s8 in range(1, 0x7F):
        e, m = s8 >> 3, s8 & 7
        d = np.float32((m * 2.0 ** -9 if e == 0 else (8 + m) * 2.0 ** (e - 10))) * ts
        for t in (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0):
            x = np.float32(d) * np.float32(t)
            near = [x]
            for _ in range(3):
                near += [np.nextafter(near[-1], np.float32(np.inf), dtype=np.float32)]
            for _ in range(3):
                near += [np.nextafter(near[0] if len(near) == 4 else near[-1], np.float32(0), dtype=np.float32)]
            rows.append([np.float32(6) * d] + near + [-v for v in near] + [np.float32(-0.0)])
    x = np.array(rows, dtype=np.float32)
    codes, sf = makepad_b200.nvfp4_quantize(ctx, torch.from_numpy(x).cuda(), float(ts))
    want_c, want_s = orc.nvfp4_quantize(x, float(ts))
    assert np.array_equal(sf.cpu().numpy(), want_s) and np.array_equal(codes.cpu().numpy(), want_c)
    if ts == 1.0:
        x = np.zeros((2, 16), dtype=np.float32)
        x[0, :4] = [np.inf, -np.inf, 100.0, -0.0]                      # the scale saturates at 448
        x[1, :4] = [np.nan, -np.nan, 12.0, -np.inf * 0]                # a NaN does not count for the scale and becomes +6
        codes, sf = makepad_b200.nvfp4_quantize(ctx, torch.from_numpy(x).cuda(), 1.0)
        assert codes[:, :2].cpu().tolist() == [[0xF7, 0x80], [0x77, 0x77]] and sf.flatten().cpu().tolist() == [0x7E, 0x40]


@pytest.mark.parametrize("M,N,K,kernel", [(1000, 4096, 14336, None), (300, 1024, 8192, None), (1, 4096, 8192, None), (257, 232, 6176, None),
                                          (1, 4096, 8192, "pair"), (16, 4096, 14336, "pair"), (64, 1024, 6176, "pair")])
def test_tiles_split_along_k(ctx, orc, monkeypatch, M, N, K, kernel):
    """Shapes whose last (or only) wave of tiles is cut along K: sampled rows against the oracle, nothing written outside the
    output, the same bits twice."""
    import torch
    import makepad_b200
    if kernel:
        monkeypatch.setenv("MPQ_FP4_KERNEL", kernel)
    a, sfa = synth.nvfp4_tensor(M, K, seed=31, stream=0)
    b, sfb = synth.nvfp4_tensor(N, K, seed=31, stream=1)
    lin = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(ctx, b, sfb, 2.0))
    ad, sd = torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda()
    buf = torch.full((M * N + 128,), 7.0, dtype=torch.bfloat16, device="cuda")
    y = buf[64:64 + M * N].view(M, N)
    lin.forward((ad, sd, 0.5), out=y)
    assert torch.equal(y, lin((ad, sd, 0.5)))
    torch.cuda.synchronize()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
    assert (buf[:64] == 7.0).all() and (buf[64 + M * N:] == 7.0).all()
    rows = sorted({0, M - 1} | set(np.random.default_rng(3).integers(0, M, 6).tolist()))
    c32, _ = orc.nvfp4_gemm(a[rows], sfa[rows], 0.5, b, sfb, 2.0)
    _check(orc, y[rows].view(torch.int16).cpu().numpy().view(np.uint16), c32)


@pytest.mark.parametrize("kernel", [None, "pair"])
def test_a_graph_of_cut_tiles_replays_after_calls_that_need_more_scratch(monkeypatch, kernel):
    """4096 x 14336: in the kernel of CTA pairs 1000 rows need 28 partial tiles, 16 rows 57 (the kernel of few rows, which takes them by default,
    cuts K in eight).  A graph of 1000 rows gives the same bits after eager calls of 16 rows and calls with another K (whose scale factors are
    re-tiled into scratch, with CTA pairs those of 64 rows too)."""
    import torch
    import makepad_b200
    if kernel:
        monkeypatch.setenv("MPQ_FP4_KERNEL", kernel)
    N, K = 4096, 14336
    c2 = makepad_b200.Context(0)
    lin = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(c2, *synth.nvfp4_tensor(N, K, seed=61, stream=1), 1.0))
    odd = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(c2, *synth.nvfp4_tensor(512, 6176, seed=62, stream=1), 1.0))
    g = torch.Generator(device="cuda")
    g.manual_seed(63)

    def rows(m, k):
        return (torch.randint(0, 256, (m, k // 2), dtype=torch.uint8, device="cuda", generator=g),
                (torch.randn((m, k // 16), device="cuda", generator=g).abs() * 0.1).to(torch.float8_e4m3fn).view(torch.uint8), 1.0)

    graphs = []
    for layer, a in ((lin, rows(1000, K)), (odd, rows(64, 6176))):
        want = layer(a)
        torch.cuda.synchronize()
        y = torch.empty_like(want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            layer.forward(a, out=y)
        graphs.append((graph, y, want, a))
    lin(rows(16, K)), odd(rows(3000, 6176))
    torch.cuda.synchronize()
    guard = [torch.full((1 << 18,), 5.0, device="cuda") for _ in range(64)]        # memory that a freed block would have become
    for graph, y, want, _ in graphs:
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    assert all((t == 5.0).all() for t in guard)
    assert c2.lib.mpq_context_poll_status(c2.h) == _lib.OK
    graphs.clear()
    c2.close()


@pytest.mark.parametrize("kernel,M", [(None, 16), ("pair", 16), (None, 70)])
@pytest.mark.parametrize("warm", ["larger", "other kernel"])
def test_a_captured_gemm_cuts_its_tiles_like_an_eager_one(orc, monkeypatch, warm, kernel, M):
    """16 and 70 rows of 4096 x 14336 want more room for partial tiles than 1000 rows do, in the kernel of CTA pairs and in the one of few rows:
    captured after a warm-up with the larger M the call still has two launches (GEMM, sum of the cut tiles) and the eager call's bits.  With
    no room reserved (the warm-up went to the one-CTA kernel) the captured call does not cut and agrees with the oracle."""
    import torch
    import makepad_b200
    N, K = 4096, 14336
    b, sfb = synth.nvfp4_tensor(N, K, seed=71, stream=1)
    a, sfa = synth.nvfp4_tensor(M, K, seed=71, stream=0)
    big = synth.nvfp4_tensor(1000, K, seed=72, stream=0)
    c2 = makepad_b200.Context(0)
    lin = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(c2, b, sfb, 1.0))
    at = (torch.from_numpy(a).cuda(), torch.from_numpy(sfa).cuda(), 0.5)
    if warm == "other kernel":
        monkeypatch.setenv("MPQ_FP4_KERNEL", "single")
    lin((torch.from_numpy(big[0]).cuda(), torch.from_numpy(big[1]).cuda(), 1.0))
    torch.cuda.synchronize()
    monkeypatch.delenv("MPQ_FP4_KERNEL", raising=False)
    if kernel:
        monkeypatch.setenv("MPQ_FP4_KERNEL", kernel)
    y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    before = c2.launches
    with torch.cuda.graph(graph):
        lin.forward(at, out=y)
    captured = c2.launches - before
    graph.replay()
    torch.cuda.synchronize()
    before = c2.launches
    eager = lin(at)
    assert c2.launches - before == 2
    assert captured == (2 if warm == "larger" else 1)
    if warm == "larger":
        assert torch.equal(y, eager)
    c32, _ = orc.nvfp4_gemm(a, sfa, 0.5, b, sfb, 1.0)
    _check(orc, y.view(torch.int16).cpu().numpy().view(np.uint16), c32)
    assert c2.lib.mpq_context_poll_status(c2.h) == _lib.OK
    del graph
    c2.close()


# Lets the next kernel in the stream start at once, then takes `ms` milliseconds (and ends in any case after 2^26 looks at the clock).
SLOW_KERNEL = r"""
extern "C" __global__ void slow_kernel(long long ms)
{
    asm volatile("griddepcontrol.launch_dependents;");
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int i = 0; i < (1 << 26); ++i) {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t - t0 > (unsigned long long)ms * 1000000ull) break;
    }
}
"""


@pytest.mark.parametrize("K", [512, 544])
def test_waits_do_not_run_out_while_earlier_kernels_are_slow(ctx, orc, K):
    """Quantisation and GEMM start beside a kernel that triggers its dependents at once and then takes a second: the GEMM's bounded
    polls begin when that has ended (K = 544: the scale factors are re-tiled by a kernel in between)."""
    import torch
    import makepad_b200
    M, N = 300, 232
    slow = torch.cuda._compile_kernel(SLOW_KERNEL, "slow_kernel")
    b, sfb = synth.nvfp4_tensor(N, K, seed=41, stream=1)
    lin = makepad_b200.QuantLinear(makepad_b200.Nvfp4Weight(ctx, b, sfb, 1.0))
    x = torch.from_numpy(synth.activations(M, K, seed=42)).cuda()
    codes, sf = makepad_b200.nvfp4_quantize(ctx, x)
    want = lin((codes, sf, 1.0))
    torch.cuda.synchronize()
    x2 = torch.zeros_like(x)
    x2.copy_(x)
    slow(grid=(1, 1, 1), block=(32, 1, 1), args=(1000,))
    codes, sf = makepad_b200.nvfp4_quantize(ctx, x2)
    y = lin((codes, sf, 1.0))
    torch.cuda.synchronize()
    assert ctx.lib.mpq_context_poll_status(ctx.h) == _lib.OK
    assert torch.equal(y, want)
