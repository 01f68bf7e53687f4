"""GPU parity of the batched-prefill paths (zc_dmmv_batch, zc_mul_mm) against the f64 oracle.

Bars: f32-activation paths relative L2 <= 1e-4 when they keep f32 precision; the bf16
tensor-core path <= 5e-3 against the exact product and <= 4e-3 against the oracle evaluated
on bf16-rounded operands (the tensor-core kernel also rounds d*sc and dmin*m to bf16 before it
forms a weight, which the rounded-operand oracle does not).
"""
import numpy as np
import pytest

import zinc_b200 as zb
from zinc_b200 import synth
from helpers import canary_intact, dev, out_with_canary, rel_l2, run_cpp

pytestmark = pytest.mark.gpu
TOL_F32, TOL_BF16, TOL_BF16_OPERANDS = 1e-4, 5e-3, 4e-3


@pytest.mark.parametrize("t", [zb.Q4_K, zb.Q6_K, zb.Q5_K, zb.Q8_0, zb.MXFP4],
                         ids=["q4_k", "q6_k", "q5_k", "q8_0", "mxfp4"])
@pytest.mark.parametrize("cols", [1, 5, 40, 129])
def test_dmmv_batch(gpu, oracle, t, cols):
    # Y[c][M] = W X[c][K]  (src/compute/dmmv.zig:880-926; layouts src/compute/forward.zig:8141-8146)
    torch, ctx, dd = gpu
    M = 96 + 7
    K = 512 if zb.block_size(t) == 256 else 160
    g = synth.rng(300, t * 1000 + cols)
    w = synth.quant_matrix(g, t, M, K)
    X = synth.activations(g, cols, K)
    Y = out_with_canary(torch, cols * M)
    dd.recordBatchDispatchPush(t, dev(torch, w), dev(torch, X), Y, M, K, 0, 0, 0, cols)
    ctx.submit_and_wait()
    got = Y[:cols * M].cpu().numpy().reshape(cols, M)
    exact = oracle.gemm_f64(w, t, M, K, X)
    assert canary_intact(Y, cols * M)
    e = rel_l2(got, exact)
    if e > TOL_F32:  # tensor-core path: compare with the bf16-operand product
        assert e <= TOL_BF16
        assert rel_l2(got, oracle.gemm_f64(w, t, M, K, X, round_bf16=True)) <= TOL_BF16_OPERANDS


@pytest.mark.parametrize("t", [zb.Q4_K, zb.Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("act", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,K", [(64, 16, 256), (300, 77, 1024), (1024, 256, 2048), (256, 300, 4096)])
def test_mul_mm(gpu, oracle, t, act, M, N, K):
    # D[col][row] = sum_k A[row][k] B[col][k], strided column-major B and D (src/compute/dmmv.zig:1045-1094)
    torch, ctx, dd = gpu
    g = synth.rng(301, t * 100 + M)
    w = synth.quant_matrix(g, t, M, K)
    Bm = synth.activations(g, N, K)
    stride_b, stride_d, b_off, d_off = K + 8, M + 4, 16, 8
    Bpad = np.zeros(b_off + N * stride_b, np.float32)
    for c in range(N):
        Bpad[b_off + c * stride_b: b_off + c * stride_b + K] = Bm[c]
    if act == "bf16":
        bits = synth.to_bf16_bits(Bpad)
        Bd = dev(torch, bits.view(np.int16))
        Bexact = synth.bf16_bits_to_f32(synth.to_bf16_bits(Bm))
    else:
        Bd = dev(torch, Bpad)
        Bexact = Bm
    D = out_with_canary(torch, d_off + N * stride_d)
    dd.recordMulMm(t, dev(torch, w), Bd, D, M, N, K, stride_b, stride_d, 0, b_off, d_off,
                   zb.BF16 if act == "bf16" else zb.F32)
    ctx.submit_and_wait()
    got = D[d_off:d_off + N * stride_d].cpu().numpy().reshape(N, stride_d)
    assert canary_intact(D, d_off + N * stride_d)
    assert np.all(got[:, M:] == 0.0), "padding between columns must stay untouched"
    exact = oracle.gemm_f64(w, t, M, K, Bexact)
    e = rel_l2(got[:, :M], exact)
    assert e <= TOL_BF16
    if e > TOL_F32:
        assert rel_l2(got[:, :M], oracle.gemm_f64(w, t, M, K, Bexact, round_bf16=True)) <= TOL_BF16_OPERANDS


@pytest.mark.parametrize("t", [zb.Q4_K, zb.Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("M,N,K", [(2043, 2600, 1024), (1280, 4100, 512), (1026, 600, 2816)])
def test_mul_mm_cta_pairs(gpu, oracle, t, M, N, K):
    """Shapes with enough tiles that K is not split and an even number of 128-row tiles: the large-tile kernel runs
    as CTA pairs (one MMA of 256 rows per pair, each CTA fetching half of every activation box). Ragged last row
    tile, a last token tile that fills one accumulator only, strided B and D."""
    torch, ctx, dd = gpu
    g = synth.rng(304, t * 100 + M)
    w = synth.quant_matrix(g, t, M, K)
    Bm = synth.activations(g, N, K)
    stride_b, stride_d = K + 8, M + 5
    Bpad = np.zeros((N, stride_b), np.float32)
    Bpad[:, :K] = Bm
    bits = synth.to_bf16_bits(Bpad.reshape(-1))
    Bexact = synth.bf16_bits_to_f32(synth.to_bf16_bits(Bm.reshape(-1))).reshape(N, K)
    D = out_with_canary(torch, N * stride_d)
    dd.recordMulMm(t, dev(torch, w), dev(torch, bits.view(np.int16)), D, M, N, K, stride_b, stride_d, 0, 0, 0, zb.BF16)
    ctx.submit_and_wait()
    got = D[:N * stride_d].cpu().numpy().reshape(N, stride_d)
    assert canary_intact(D, N * stride_d)
    assert np.all(got[:, M:] == 0.0), "padding between columns must stay untouched"
    exact = oracle.gemm_f64(w, t, M, K, Bexact)
    assert rel_l2(got[:, :M], exact) <= TOL_BF16
    assert rel_l2(got[:, :M], oracle.gemm_f64(w, t, M, K, Bexact, round_bf16=True)) <= TOL_BF16_OPERANDS
    # every row tile against its own rows: a pair that swapped or dropped a half would pass no global norm
    for r0 in range(0, M, 128):
        assert rel_l2(got[:, r0:min(r0 + 128, M)], exact[:, r0:r0 + 128]) <= TOL_BF16
    for c0 in range(0, N, 128):
        assert rel_l2(got[c0:c0 + 128, :M], exact[c0:c0 + 128]) <= TOL_BF16


@pytest.mark.parametrize("M,N,K", [(2048, 1100, 6144), (512, 700, 2048)], ids=["flags", "zeroed"])
def test_mul_mm_cta_pairs_recorded(gpu, oracle, M, N, K):
    """The pair kernel inside a recording, replayed. Tiles split over pairs are summed through memory: with long
    ranges (24 tiles x 24 blocks over 74 pairs) behind per-tile flags that a memset node of the recording clears (a
    flag left up would let an adder run ahead of the stores it adds to, a flag left down would time out), with
    short ranges (4 tiles x 8 blocks over 8 pairs) by adding into D, which a memset node zeroes. Either way every
    replay has to give the product again."""
    torch, _, _ = gpu
    t = zb.Q4_K
    g = synth.rng(305, 1)
    w = synth.quant_matrix(g, t, M, K)
    Bm = synth.activations(g, N, K)
    bits = synth.to_bf16_bits(Bm.reshape(-1))
    Bexact = synth.bf16_bits_to_f32(bits).reshape(N, K)
    exact = oracle.gemm_f64(w, t, M, K, Bexact)
    stream = torch.cuda.Stream()   # a stream of its own: the default stream cannot be captured
    with torch.cuda.stream(stream):
        ctx = zb.Context(0, stream=stream.cuda_stream)
        dd = zb.DmmvDispatch(ctx)
        wd, bd = dev(torch, w), dev(torch, bits.view(np.int16))
        D = out_with_canary(torch, N * M)
        stream.synchronize()
        ctx.begin_record()
        dd.recordMulMm(t, wd, bd, D, M, N, K, K, M, 0, 0, 0, zb.BF16)
        rec = ctx.end_record()
        try:
            for _ in range(3):
                D[:N * M] = float("nan")
                ctx.replay(rec)
                ctx.submit_and_wait()
                got = D[:N * M].cpu().numpy().reshape(N, M)
                assert canary_intact(D, N * M)
                assert rel_l2(got, exact) <= TOL_BF16
        finally:
            ctx.free_recording(rec)


@pytest.mark.parametrize("M,N,K", [(64, 16, 64), (300, 77, 320), (200, 32, 2880), (256, 300, 2880),
                                   (1000, 700, 2880), (1152, 520, 448)])
def test_mul_mm_mxfp4_bf16(gpu, oracle, M, N, K):
    # MXFP4 weights dequantise exactly to bf16, so with bf16 activations the tensor-core product differs
    # from the exact one only by the f32 accumulation order (rows of 17-byte blocks: no alignment at all)
    torch, ctx, dd = gpu
    t = zb.MXFP4
    g = synth.rng(302, M + K)
    w = synth.quant_matrix(g, t, M, K)
    Bm = synth.activations(g, N, K)
    bits = synth.to_bf16_bits(Bm.reshape(-1))
    Bexact = synth.bf16_bits_to_f32(bits).reshape(N, K)
    D = out_with_canary(torch, N * M)
    dd.recordMulMm(t, dev(torch, w), dev(torch, bits.view(np.int16)), D, M, N, K, K, M, 0, 0, 0, zb.BF16)
    ctx.submit_and_wait()
    got = D[:N * M].cpu().numpy().reshape(N, M)
    assert canary_intact(D, N * M)
    assert rel_l2(got, oracle.gemm_f64(w, t, M, K, Bexact)) <= 1e-5


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (256, 128, 512), (300, 200, 2880), (1024, 600, 2880), (130, 64, 160)])
def test_mul_mm_mxfp4_block_scaled(gpu, oracle, M, N, K):
    """MXFP4 weights as stored on the block-scaled tensor-core path (zc_mul_mm_block_scaled): the two FP8 terms add
    up to the bf16 activation exactly, so the product differs from the exact one by the f32 accumulation only.
    Row, token and K counts that are not multiples of the tile, a wide activation range inside a block, and the
    launch count (split + GEMM) that shows this path ran."""
    torch, ctx, dd = gpu
    t = zb.MXFP4
    g = synth.rng(303, M + K + N)
    w = synth.quant_matrix(g, t, M, K)
    Bm = synth.activations(g, N, K)
    Bm[:, ::7] *= np.float32(64.0)      # spread of magnitudes inside a 32-element block
    Bm[:, 3::11] *= np.float32(1.0 / 128.0)
    Bm[N // 2, :32] = 0.0               # an all-zero block
    bits = synth.to_bf16_bits(Bm.reshape(-1))
    Bexact = synth.bf16_bits_to_f32(bits).reshape(N, K)
    D = out_with_canary(torch, N * M)
    ws = torch.empty(dd.mulMmWorkspaceBytes(t, N, K), dtype=torch.uint8, device="cuda")
    assert ws.numel() > 0 and dd.mulMmWorkspaceBytes(zb.Q4_K, N, K) == 0
    n0 = ctx.launch_count
    dd.recordMulMmBlockScaled(t, dev(torch, w), dev(torch, bits.view(np.int16)), D, M, N, K, K, M, ws)
    ctx.submit_and_wait()
    assert ctx.launch_count - n0 == 2
    with pytest.raises(zb.InvalidArgument):   # a workspace that is too small
        dd.recordMulMmBlockScaled(t, dev(torch, w), dev(torch, bits.view(np.int16)), D, M, N, K, K, M, ws[:1024])
    with pytest.raises(zb.UnsupportedQuantType):
        dd.recordMulMmBlockScaled(zb.Q4_K, dev(torch, w), dev(torch, bits.view(np.int16)), D, M, N, K, K, M, ws)
    got = D[:N * M].cpu().numpy().reshape(N, M)
    assert canary_intact(D, N * M)
    assert rel_l2(got, oracle.gemm_f64(w, t, M, K, Bexact)) <= 1e-5


# Relative L2 of the f32-accurate GEMM: 2^-23 for an activation of two fp16 terms, at most 34 tensor-core accumulations
# of a block and K / 256 f32 additions of 2^-23 each in the worst case, their random sum in practice.
TOL_EXACT = 5e-6


@pytest.mark.parametrize("t,act", [(zb.Q4_K, "f32"), (zb.Q5_K, "f32"), (zb.Q5_K, "bf16"), (zb.Q6_K, "f32"), (zb.Q8_0, "f32"),
                                   (zb.Q8_0, "bf16"), (zb.MXFP4, "f32")])
@pytest.mark.parametrize("M,N,K", [(1, 2, 256), (129, 33, 256), (257, 64, 512), (300, 65, 2048), (127, 129, 768),
                                   (520, 257, 1024), (2050, 17, 2304), (256, 600, 512), (100, 40, 160)])
def test_mul_mm_exact(gpu, oracle, t, act, M, N, K):
    """Tile edges in rows and tokens (32, 64, 128, 256), one block, whole and split tiles, block tails past K, rows with
    and without a 16-byte pitch."""
    torch, ctx, dd = gpu
    if K % zb.block_size(t):
        K = 256
    g = synth.rng(305, t * 100 + M + N)
    w = synth.quant_matrix(g, t, M, K)
    # tokens of very different magnitude: each has a scale of its own
    X = (synth.activations(g, N, K) * np.exp2(np.arange(N) % 40 - 20)[:, None]).astype(np.float32)
    if act == "bf16":
        bits = synth.to_bf16_bits(X)
        Xd, X = dev(torch, bits.view(np.int16)), synth.bf16_bits_to_f32(bits)
    else:
        Xd = dev(torch, X)
    D = out_with_canary(torch, N * M, init=7.0)
    wd = dev(torch, w)
    for _ in range(2):   # the second call finds the context's scratch as the first one left it
        dd.recordMulMm(t, wd, Xd, D, M, N, K, K, M, act_type=zb.BF16 if act == "bf16" else zb.F32)
    ctx.submit_and_wait()
    got = D[:N * M].cpu().numpy().reshape(N, M)
    want = oracle.gemm_f64(w, t, M, K, X)
    assert canary_intact(D, N * M)
    for c in range(N):
        assert rel_l2(got[c], want[c]) <= (TOL_EXACT if M > 1 else 50 * TOL_EXACT)   # M = 1: one value, cancellation


@pytest.mark.parametrize("t,act", [(zb.Q4_K, "f32"), (zb.Q5_K, "bf16"), (zb.Q6_K, "f32"), (zb.Q8_0, "bf16"), (zb.MXFP4, "f32")])
@pytest.mark.parametrize("M,N,K", [(5000, 145, 768), (5000, 209, 768), (4400, 193, 2048), (9000, 257, 512), (9000, 481, 512),
                                   (9000, 700, 512)])
def test_mul_mm_exact_tile_widths(gpu, oracle, t, act, M, N, K):
    """Tiles of 48 to 256 tokens that are no multiples of 32, of both splits of the warps (to 192 tokens and beyond), raw
    blocks by TMA and fetched."""
    torch, ctx, dd = gpu
    g = synth.rng(311, t * 100 + M + N)
    w = synth.quant_matrix(g, t, M, K)
    X = synth.activations(g, N, K)
    if act == "bf16":
        bits = synth.to_bf16_bits(X)
        Xd, X = dev(torch, bits.view(np.int16)), synth.bf16_bits_to_f32(bits)
    else:
        Xd = dev(torch, X)
    D = out_with_canary(torch, N * M, init=7.0)
    dd.recordMulMm(t, dev(torch, w), Xd, D, M, N, K, K, M, act_type=zb.BF16 if act == "bf16" else zb.F32)
    ctx.submit_and_wait()
    got = D[:N * M].cpu().numpy().reshape(N, M)
    assert canary_intact(D, N * M)
    want = oracle.gemm_f64(w, t, M, K, X)
    for c in range(N):
        assert rel_l2(got[c], want[c]) <= TOL_EXACT


@pytest.mark.parametrize("t", [zb.Q4_K, zb.Q5_K], ids=["q4_k", "q5_k"])
def test_mul_mm_exact_scale_ratios(gpu, oracle, t):
    """Blocks whose d and dmin lie far apart: d = 0, dmin = 0, dmin / d from 2^-14 to 2^17, negative scales."""
    torch, ctx, dd = gpu
    M, N, K = 64, 20, 512
    g = synth.rng(306, t)
    w = synth.quant_matrix(g, t, M, K).reshape(M * 2, -1)
    d = np.exp2(-(np.arange(M * 2) % 12)).astype(np.float16) * np.where(np.arange(M * 2) % 5 == 0, -1, 1).astype(np.float16)
    dmin = np.exp2(np.arange(M * 2) % 17 - 10).astype(np.float16)
    d[:4], dmin[4:8] = 0, 0
    d[8:12], dmin[8:12] = np.float16(2.0 ** -14), np.float16(8.0)   # 2^17: both go down by powers of two
    w[:, 0:2], w[:, 2:4] = d.view(np.uint8).reshape(-1, 2), dmin.view(np.uint8).reshape(-1, 2)
    X = synth.activations(g, N, K)
    D = out_with_canary(torch, N * M)
    dd.recordMulMm(t, dev(torch, w.reshape(-1)), dev(torch, X), D, M, N, K, K, M)
    ctx.submit_and_wait()
    got = D[:N * M].cpu().numpy().reshape(N, M)
    want = oracle.gemm_f64(w.reshape(-1), t, M, K, X)
    for r in range(M):
        assert rel_l2(got[:, r], want[:, r]) <= 2 * TOL_EXACT


@pytest.mark.parametrize("t", [zb.Q4_K, zb.Q5_K, zb.Q6_K, zb.Q8_0, zb.MXFP4], ids=["q4_k", "q5_k", "q6_k", "q8_0", "mxfp4"])
@pytest.mark.parametrize("cols", [7, 64, 65, 130])
def test_dmmv_batch_is_as_accurate_as_f32_sums(gpu, oracle, t, cols):
    """The batched product on the tensor cores against f64. Bound, relative L2: 1.2e-7 for the four truncations of a
    64-column run (half of 2^-23 each, the partial sums before the last one smaller), 1.7e-7 for the 64 f32 additions of
    4096 columns (0.29 x 2^-23 each, as a random sum), 0.5e-7 for activations of 22 bits: 2.1e-7 together, some 20 % to
    spare. (Accumulations of 256 columns have 3.6e-7 and more.)"""
    torch, ctx, dd = gpu
    M, K = 512, 4096
    g = synth.rng(310, t + cols)
    w = synth.quant_matrix(g, t, M, K)
    X = synth.activations(g, cols, K)
    Y = out_with_canary(torch, cols * M)
    dd.recordBatchDispatchPush(t, dev(torch, w), dev(torch, X), Y, M, K, 0, 0, 0, cols)
    ctx.submit_and_wait()
    assert canary_intact(Y, cols * M)
    assert rel_l2(Y[:cols * M].cpu().numpy(), oracle.gemm_f64(w, t, M, K, X)) <= 2.5e-7


@pytest.mark.parametrize("t", [zb.Q4_K, zb.Q5_K, zb.Q6_K, zb.Q8_0, zb.MXFP4], ids=["q4_k", "q5_k", "q6_k", "q8_0", "mxfp4"])
@pytest.mark.parametrize("N", [20, 150])
def test_mul_mm_exact_outlier_inside_a_token(gpu, oracle, t, N):
    """One element of a token 2^16 above the others, against weights that are zero: the others, 2^-16 of the largest or a
    little less, keep their 22 bits, so that the bound is the one of tokens without outliers."""
    torch, ctx, dd = gpu
    M, K = 70, 1024
    g = synth.rng(308, t)
    w = synth.quant_matrix(g, t, M, K).reshape(M, -1).copy()
    one = zb.row_bytes(t, 256)
    w[:, one:2 * one] = 0   # columns 256 .. 511
    X = synth.activations(g, N, K)
    X[:, 300] = np.where(np.arange(N) % 2, -65536.0, 65536.0).astype(np.float32)
    D = out_with_canary(torch, N * M)
    dd.recordMulMm(t, dev(torch, w.reshape(-1)), dev(torch, X), D, M, N, K, K, M)
    ctx.submit_and_wait()
    want = oracle.gemm_f64(w.reshape(-1), t, M, K, X)
    got = D[:N * M].cpu().numpy().reshape(N, M)
    for c in range(N):
        assert rel_l2(got[c], want[c]) <= TOL_EXACT


def test_mul_mm_exact_wide_block_scales(gpu, oracle):
    """Scales within 256 columns far apart. MXFP4: 2^-20 of the largest, whose block holds zeros: exact. Q8_0: d 2^-12 of the
    largest: exact. Q4_K: dmin 2^20 times d against mins that cancel: the q terms still count in full."""
    torch, ctx, dd = gpu
    M, N, K = 40, 24, 256
    g = synth.rng(309, 0)
    X = synth.activations(g, N, K)

    def run(t, w, X):
        D = out_with_canary(torch, N * M)
        dd.recordMulMm(t, dev(torch, w.reshape(-1)), dev(torch, X), D, M, N, K, K, M)
        ctx.submit_and_wait()
        return D[:N * M].cpu().numpy().reshape(N, M), oracle.gemm_f64(np.ascontiguousarray(w).reshape(-1), t, M, K, X)

    w = synth.quant_matrix(g, zb.MXFP4, M, K).reshape(M, 8, 17).copy()
    w[:, :, 0] = 110
    w[:, 3, 0], w[:, 3, 1:] = 130, 0
    got, want = run(zb.MXFP4, w, X)
    assert rel_l2(got, want) <= TOL_EXACT
    w = synth.quant_matrix(g, zb.Q8_0, M, K).reshape(M, 8, 34).copy()
    w[:, :, 0:2] = np.frombuffer(np.float16(2.0 ** -12 * 1.25).tobytes(), np.uint8)
    w[:, 5, 0:2], w[:, 5, 2:] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8), 0
    got, want = run(zb.Q8_0, w, X)
    assert rel_l2(got, want) <= TOL_EXACT
    w = synth.quant_matrix(g, zb.Q4_K, M, K).reshape(M, 144).copy()
    w[:, 0:2] = np.frombuffer(np.float16(2.0 ** -17).tobytes(), np.uint8)
    w[:, 2:4] = np.frombuffer(np.float16(8.0).tobytes(), np.uint8)
    Xz = X.copy()
    Xz[:, 1::2] = -Xz[:, ::2]   # every sub-block sums to zero: the min terms vanish, exactly
    got, _ = run(zb.Q4_K, w, Xz)
    w[:, 2:4] = 0               # (a weight dequantised to one f32 would have lost its q term beside the min)
    assert rel_l2(got, oracle.gemm_f64(np.ascontiguousarray(w).reshape(-1), zb.Q4_K, M, K, Xz)) <= TOL_EXACT


@pytest.mark.parametrize("t,K", [(zb.Q6_K, 2048), (zb.Q8_0, 2048), (zb.MXFP4, 2080)], ids=["q6_k", "q8_0", "mxfp4"])
def test_mul_mm_exact_same_bits_every_time(gpu, t, K):
    """A raw slot given back while a read of it is under way changes single rows now and then; a repeated launch has to
    give the same bits. (74 whole tiles: no sum has two writers.)"""
    torch, ctx, dd = gpu
    M, N = 256 * 37, 512
    g = synth.rng(307, t)
    w, X = dev(torch, synth.quant_matrix(g, t, M, K)), dev(torch, synth.activations(g, N, K))
    first, bad = None, 0
    for _ in range(300):
        D = torch.empty(N * M, device="cuda")
        dd.recordMulMm(t, w, X, D, M, N, K, K, M)
        first = D if first is None else first
        bad = bad + (D != first).sum()
    ctx.submit_and_wait()
    assert int(bad) == 0


@pytest.mark.parametrize("t,M,N,K,bf16", [(t, *s, False) for t in (zb.Q4_K, zb.Q6_K, zb.MXFP4) for s in
                                          ((300, 5, 8192), (1027, 41, 3840), (4096, 64, 4096), (2048, 256, 8192), (4096, 658, 4096))] +
                         [(zb.Q6_K, 1027, 41, 3840, True), (zb.Q6_K, 4096, 64, 11008, True), (zb.MXFP4, 1027, 41, 3840, True),
                          (zb.MXFP4, 300, 200, 8192, True)])
def test_split_gemm_is_reproducible(gpu, oracle, t, M, N, K, bf16):
    """Few tiles, which K is split for: f32 activations over CTA pairs, bf16 where rows have no pitch of 16 bytes over CTAs.
    The same bits every time and the right sums (f32: 2e-6, above the 1.1e-6 of one f32 chain per output; rows past M, tokens
    past N)."""
    torch, ctx, dd = gpu
    g = synth.rng(317, M + N + t)
    raw, X = synth.quant_matrix(g, t, M, K), synth.activations(g, N, K)
    w, x = dev(torch, raw), dev(torch, X)
    if bf16:
        x = x.to(torch.bfloat16)
        X = x.float().cpu().numpy()
    first = None
    for i in range(12):
        D = torch.full((N + 1, M), 7.0, device="cuda")
        torch.cuda.synchronize()
        dd.recordMulMm(t, w, x, D, M, N, K, K, M, act_type=zb.BF16 if bf16 else zb.F32)
        ctx.submit_and_wait()
        got = D.cpu()
        if first is None:
            first = got
        assert torch.equal(got, first)
    assert (first[N:] == 7.0).all()
    cols = sorted({0, N // 2, N - 1})
    assert rel_l2(first[cols].numpy(), oracle.gemm_f64(raw, t, M, K, X[cols])) <= (TOL_BF16 if bf16 else 2e-6)


def test_mul_mm_cut_in_every_form(gpu):
    """Every number of CTAs and every cluster that K can be cut over, and waits that run out, with copies and MMAs under way."""
    run_cpp("test_cut")


# Shapes that the rule cuts K of over 1, 2, 4, 6, 8, 10 and 16 CTAs (148 SMs; every form by itself: the test above); tokens on both sides
# of a tile's 192 and of 16, one block of K, rows on both sides of 8 and 128 (Q6_K: boxes of every eighth row), rows of D that start
# anywhere and at 16 bytes only
@pytest.mark.parametrize("t,M,N,K", [(t, *s) for t in (zb.Q4_K, zb.Q6_K) for s in
                                     ((1, 16, 256), (127, 17, 512), (130, 192, 1024), (263, 193, 2560), (1024, 77, 4096), (1027, 385, 768),
                                      (300, 40, 11520), (641, 209, 3328), (2050, 31, 1280), (515, 1500, 256),
                                      (1743, 378, 3072), (1152, 130, 2560))])
@pytest.mark.parametrize("pad_b,pad_d,d_off", [(0, 0, 0), (8, 3, 1), (24, 4, 4)])
def test_mul_mm_cut(gpu, oracle, t, M, N, K, pad_b, pad_d, d_off):
    torch, ctx, dd = gpu
    g = synth.rng(341, M + N + t)
    raw, X = synth.quant_matrix(g, t, M, K), synth.activations(g, N, K)
    X = synth.bf16_bits_to_f32(synth.to_bf16_bits(X))
    Xp = np.zeros((N, K + pad_b), np.float32)
    Xp[:, :K] = X
    w, x = dev(torch, raw), dev(torch, Xp).to(torch.bfloat16)
    first = None
    for i in range(4):
        D = torch.full((d_off + (N + 1) * (M + pad_d),), 7.0, device="cuda")
        torch.cuda.synchronize()
        dd.recordMulMm(t, w, x, D, M, N, K, K + pad_b, M + pad_d, 0, 0, d_off, zb.BF16)
        ctx.submit_and_wait()
        got = D.cpu()
        first = got if first is None else first
        assert torch.equal(got, first), "not the same bits"
    assert (first[:d_off] == 7.0).all()
    first = first[d_off:].view(N + 1, M + pad_d)
    assert (first[N:] == 7.0).all() and (first[:, M:] == 7.0).all()
    cols = sorted({0, 15, N // 2, N - 1})
    assert rel_l2(first[cols, :M].numpy(), oracle.gemm_f64(raw, t, M, K, X[cols], round_bf16=True)) <= TOL_BF16_OPERANDS


@pytest.mark.parametrize("t,M,N,K,bf16,want", [
    (zb.Q4_K, 256, 40, 4096, True, 2),      # K split: zeroing kernel, GEMM
    (zb.Q4_K, 40960, 40, 256, True, 1),
    (zb.Q6_K, 256, 200, 4096, True, 2),
    (zb.Q4_K, 1024, 600, 4096, True, 2),    # CTA pairs: D or the tiles' flags zeroed, GEMM
    (zb.MXFP4, 256, 40, 1024, True, 2),     # two slices of K: zeroing kernel, GEMM
    (zb.MXFP4, 256, 40, 4096, True, 2),     # eight: GEMM, sums of the parts
    (zb.Q4_K, 256, 40, 4096, False, 3),     # preparation, GEMM, sums of the parts
    (zb.Q4_K, 20480, 40, 256, False, 2)])
def test_mul_mm_counts_its_launches(gpu, t, M, N, K, bf16, want):
    torch, ctx, dd = gpu
    g = synth.rng(337, M)
    w, x = dev(torch, synth.quant_matrix(g, t, M, K)), dev(torch, synth.activations(g, N, K))
    D = torch.empty(N, M, device="cuda")
    before = ctx.launch_count
    dd.recordMulMm(t, w, x.to(torch.bfloat16) if bf16 else x, D, M, N, K, K, M, act_type=zb.BF16 if bf16 else zb.F32)
    assert ctx.launch_count - before == want
    ctx.submit_and_wait()


@pytest.mark.parametrize("t,M,N,K,bf16", [(zb.Q4_K, 20480, 32, 256, True), (zb.Q6_K, 10240, 32, 2048, True), (zb.Q4_K, 10240, 200, 256, True),
                                          (zb.MXFP4, 20480, 32, 64, True), (zb.Q4_K, 4096, 40, 256, False)])
def test_mul_mm_reads_weights_of_the_kernel_before(gpu, t, M, N, K, bf16):
    """Weights that the kernel directly in front on the stream writes (shapes without a zeroing kernel between them too)."""
    torch, _, _ = gpu
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = zb.Context(0, stream=stream.cuda_stream)
        dd = zb.DmmvDispatch(ctx)
        g = synth.rng(331, M + N)
        W = [dev(torch, synth.quant_matrix(g, t, M, K)) for _ in range(2)]
        x = dev(torch, synth.activations(g, N, K))
        x = x.to(torch.bfloat16) if bf16 else x
        w = torch.empty_like(W[0])
        D = [torch.empty(N, M, device="cuda") for _ in range(10)]
        for i in range(10):
            if i < 2:
                torch.cuda.synchronize()
            w.copy_(W[i % 2])
            w.bitwise_or_(0)  # a kernel
            if i < 2:
                torch.cuda.synchronize()
            dd.recordMulMm(t, w, x, D[i], M, N, K, K, M, act_type=zb.BF16 if bf16 else zb.F32)
        ctx.submit_and_wait()
        for i in range(2, 10):
            assert torch.equal(D[i], D[i % 2])
        assert not torch.equal(D[0], D[1])
        ctx.close()


def test_mul_mm_exact_on_two_streams(gpu):
    """The f32-accurate GEMM keeps the terms of its activations in the context's scratch: a call on another stream, or a
    replay there, may not overwrite what a call still under way reads."""
    torch, _, _ = gpu
    M, N, K, n = 2048, 300, 2048, 24
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    ctx = zb.Context(0, stream=s1.cuda_stream)
    dd = zb.DmmvDispatch(ctx)
    g = synth.rng(311, 0)
    w = dev(torch, synth.quant_matrix(g, zb.Q4_K, M, K))
    X = [dev(torch, synth.activations(g, N, K)) for _ in range(4)]
    want = []
    for x in X:
        D = torch.empty(N, M, device="cuda")
        torch.cuda.synchronize()
        dd.recordMulMm(zb.Q4_K, w, x, D, M, N, K, K, M)
        ctx.submit_and_wait()
        want.append(D)
    Y = torch.empty(N, M, device="cuda")
    ctx.begin_record()
    dd.recordMulMm(zb.Q4_K, w, X[3], Y, M, N, K, K, M)
    recording = ctx.end_record()
    got = [torch.empty(N, M, device="cuda") for _ in range(n)]
    torch.cuda.synchronize()
    for i in range(n):
        ctx.set_stream((s1, s2)[i % 2].cuda_stream)
        if i % 5 == 4:
            ctx.replay(recording)
        else:
            dd.recordMulMm(zb.Q4_K, w, X[i % 3], got[i], M, N, K, K, M)
    torch.cuda.synchronize()
    ctx.submit_and_wait()
    for i in range(n):
        if i % 5 != 4:
            assert float((got[i] - want[i % 3]).norm() / want[i % 3].norm()) <= 1e-6
    assert float((Y - want[3]).norm() / want[3].norm()) <= 1e-6
    ctx.free_recording(recording)
    ctx.close()


def test_mul_mm_errors(gpu):
    torch, ctx, dd = gpu
    w = torch.zeros(144 * 8, dtype=torch.uint8, device="cuda")
    b = torch.zeros(4 * 256, device="cuda")
    d = torch.zeros(4 * 8, device="cuda")
    with pytest.raises(zb.InvalidArgument):  # K misaligned (src/compute/dmmv.zig:1065)
        dd.recordMulMmQ4K(w, b, d, 8, 4, 200, 256, 8)
    with pytest.raises(zb.InvalidArgument):  # N == 0 (src/compute/dmmv.zig:1066)
        dd.recordMulMmQ4K(w, b, d, 8, 0, 256, 256, 8)
    with pytest.raises(zb.UnsupportedQuantType):
        dd.recordMulMm(11, w, b, d, 8, 4, 256, 256, 8)
    dd.recordMulMmQ4K(w, b, d, 8, 4, 256, 256, 8)
    ctx.submit_and_wait()
