"""Parity of the CUDA GEMMLowp path (through the C ABI) with the oracle: bit-exact, tolerance 0."""
import os

import numpy as np
import pytest

from computelibrary_b200 import capi
from helpers import (golden_int_stage, config1, config2, config5, f32_mults, golden_gemm_cases, gpu_gemmlowp, q8_uniform, type_range)

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


@pytest.fixture(scope="module")
def gemm_golden():
    return np.load(os.path.join(GOLDEN, "gemmlowp_golden.npz"))


@pytest.mark.parametrize("force_simt", [False, True])
def test_golden_cases(ctx, gemm_golden, force_simt):
    """Reference-produced outputs on odd shapes (M=1, N=1, K not a multiple of 16): S32 core, per-tensor and
    per-channel fused output stage, for u8xu8, s8xs8 and u8xs8."""
    for g in golden_gemm_cases():
        acc, _ = gpu_gemmlowp(ctx, g["a"], g["b"], None, g["a_off"], g["b_off"], 0, 0, 0, 0, 0, np.int32,
                              force_simt=force_simt)
        assert np.array_equal(acc, gemm_golden[g["key"] + "_acc"]), g["key"]
        pt, _ = gpu_gemmlowp(ctx, g["a"], g["b"], g["bias"], g["a_off"], g["b_off"], int(g["mult"][0]),
                             int(g["shift"][0]), g["pt_offset"], g["lo"], g["hi"], g["out_dtype"],
                             force_simt=force_simt)
        assert np.array_equal(pt, gemm_golden[g["key"] + "_pt"]), g["key"]
        pc, _ = gpu_gemmlowp(ctx, g["a"], g["b"], g["bias"], g["a_off"], 0, g["mult"], g["shift"], g["pc_offset"],
                             g["lo"], g["hi"], g["out_dtype"], force_simt=force_simt)
        assert np.array_equal(pc, gemm_golden[g["key"] + "_pc"]), g["key"]


def test_config1_fused_and_two_stage(ctx, port, gemm_golden):
    """Configuration 1 of the benchmark against the reference-produced fixture, fused and as core(S32) + output stage."""
    import torch
    c1 = config1()
    qm, sh = capi.calculate_quantized_multiplier(c1["real_multiplier"])
    assert (qm, sh) == (1099511552, 8)
    out, kernel = gpu_gemmlowp(ctx, c1["a"], c1["b"], c1["bias"], c1["a_off"], c1["b_off"], qm, sh, c1["offset"],
                               c1["lo"], c1["hi"], np.uint8)
    assert kernel == "tcgen05"  # 64 rows: one CTA per tile
    assert np.array_equal(out, gemm_golden["c1_out"])
    acc, _ = gpu_gemmlowp(ctx, c1["a"], c1["b"], None, c1["a_off"], c1["b_off"], 0, 0, 0, 0, 0, np.int32)
    assert np.array_equal(acc, gemm_golden["c1_acc"])
    # NEGEMMLowpOutputStage on the S32 result (examples/neon_gemm_qasymm8.cpp:224-239)
    d_acc = torch.from_numpy(acc).cuda()
    d_bias = torch.from_numpy(c1["bias"]).cuda()
    d_out = torch.empty((64, 128), dtype=torch.uint8, device="cuda")
    ctx.output_stage(d_acc, 128 * 4, d_bias, d_out, 128, capi.U8, 64, 128, None, None, qm, sh, 1, c1["offset"],
                     c1["lo"], c1["hi"])
    ctx.sync()
    assert np.array_equal(d_out.cpu().numpy(), gemm_golden["c1_out"])
    # as-given (non-negated) offsets are part of the contract too
    out2, _ = gpu_gemmlowp(ctx, c1["a"], c1["b"], c1["bias"], 128, 120, qm, sh, c1["offset"], 0, 255, np.uint8)
    want2 = port.gemmlowp_fused(c1["a"], c1["b"], c1["bias"], 128, 120, [qm], [sh], c1["offset"], 0, 255, np.uint8)
    assert np.array_equal(out2, want2)


SHAPES = [(128, 256, 128), (129, 257, 130), (64, 64, 16), (300, 520, 1000), (1, 1000, 2048), (257, 64, 576),
          (1000, 96, 147), (512, 128, 4608), (37, 1, 5)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("types", ["u8u8", "s8s8", "u8s8"])
def test_fused_vs_oracle(ctx, port, M, N, K, types):
    ad = np.uint8 if types[:2] == "u8" else np.int8
    bd = np.uint8 if types[2:] == "u8" else np.int8
    rng = np.random.default_rng(M * 131 + N * 17 + K)
    a, b = q8_uniform(rng, (M, K), ad), q8_uniform(rng, (K, N), bd)
    bias = rng.integers(-5000, 5001, N).astype(np.int32)
    lo, hi = type_range(ad)
    # per-tensor, both offsets
    ao, bo = int(rng.integers(-200, 200)), int(rng.integers(-200, 200))
    qm, sh = capi.calculate_quantized_multiplier(np.float32(3.0 / (K * 40.0)))
    want = port.gemmlowp_fused(a, b, bias, ao, bo, [qm], [sh], 7, lo, hi, ad)
    for simt, pair in ((False, True), (False, False), (True, True)):  # SM-pair, one-CTA and generic kernels
        got, kern = gpu_gemmlowp(ctx, a, b, bias, ao, bo, qm, sh, 7, lo, hi, ad, force_simt=simt, ldd_pad=16,
                                 pair=pair)
        assert np.array_equal(got, want), (kern, np.argwhere(got != want)[:5])
    # per-channel (b_offset 0), log-uniform scales as in the benchmark configs
    ws = np.exp(rng.uniform(np.log(1e-3), np.log(1e-2), N)).astype(np.float32)
    mult, shift = f32_mults(port, 0.02, ws, 0.02 * 0.005 * K * 30)
    got, kern = gpu_gemmlowp(ctx, a, b, bias, ao, 0, mult, shift, -3, lo + 2, hi - 3, ad)
    want = port.gemmlowp_fused(a, b, bias, ao, 0, mult, shift, -3, lo + 2, hi - 3, ad)
    assert np.array_equal(got, want), kern
    # S32 core
    got, _ = gpu_gemmlowp(ctx, a, b, None, ao, bo, 0, 0, 0, 0, 0, np.int32, ldd_pad=4)
    assert np.array_equal(got, port.gemmlowp_core(a, b, ao, bo))


def test_kernel_selection(ctx):
    rng = np.random.default_rng(0)
    a, b = q8_uniform(rng, (64, 48), np.uint8), q8_uniform(rng, (48, 32), np.uint8)
    _, k1 = gpu_gemmlowp(ctx, a, b, None, 0, 0, 2 ** 30, 3, 0, 0, 255, np.uint8)
    assert k1 == "tcgen05"          # K = 48: row stride is a multiple of 16 bytes
    a2, b2 = q8_uniform(rng, (64, 50), np.uint8), q8_uniform(rng, (50, 32), np.uint8)
    got, k2 = gpu_gemmlowp(ctx, a2, b2, None, 0, 0, 2 ** 30, 3, 0, 0, 255, np.uint8)
    # K = 50: TMA cannot address these rows of A, so the plan multiplies a copy of A with a 64-byte row pitch
    assert k2 == "tcgen05"
    _, k3 = gpu_gemmlowp(ctx, a2, b2, None, 0, 0, 2 ** 30, 3, 0, 0, 255, np.uint8, force_simt=True)
    assert k3 == "simt" and np.array_equal(got, _)


def test_negative_shift_and_saturating_multiplier(ctx, port):
    """Left shifts (multiplier >= 1) and the INT32_MIN * INT32_MIN corner of SQDMULH."""
    rng = np.random.default_rng(2)
    M, N, K = 130, 70, 64
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, N), np.int8)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
    shift = rng.integers(-3, 4, N).astype(np.int32)
    mult[5] = -2 ** 31
    bias = rng.integers(-100, 100, N).astype(np.int32)
    for simt in (False, True):
        got, _ = gpu_gemmlowp(ctx, a, b, bias, 3, 0, mult, shift, 1, -128, 127, np.int8, force_simt=simt)
        assert np.array_equal(got, port.gemmlowp_fused(a, b, bias, 3, 0, mult, shift, 1, -128, 127, np.int8))
    qm, sh = capi.calculate_quantized_multiplier(np.float32(2.5))
    assert sh < 0
    got, _ = gpu_gemmlowp(ctx, a, b, None, 0, 0, qm, sh, 0, -128, 127, np.int8)
    assert np.array_equal(got, port.gemmlowp_fused(a, b, None, 0, 0, [qm], [sh], 0, -128, 127, np.int8))


def test_batched(ctx, port):
    """BatchedMatMul (tests/validation/NEON/GEMMLowp.cpp:317-359): batched A with shared and batched B."""
    rng = np.random.default_rng(4)
    a = q8_uniform(rng, (3, 70, 96), np.int8)
    b1 = q8_uniform(rng, (96, 40), np.int8)
    b3 = q8_uniform(rng, (3, 96, 40), np.int8)
    qm, sh = capi.calculate_quantized_multiplier(np.float32(0.0007))
    for b in (b1, b3):
        got, _ = gpu_gemmlowp(ctx, a, b, None, 4, -6, qm, sh, 2, -128, 127, np.int8)
        for i in range(3):
            bi = b if b.ndim == 2 else b[i]
            want = port.gemmlowp_fused(a[i], bi, None, 4, -6, [qm], [sh], 2, -128, 127, np.int8)
            assert np.array_equal(got[i], want)
        acc, _ = gpu_gemmlowp(ctx, a, b, None, 4, -6, 0, 0, 0, 0, 0, np.int32)
        assert np.array_equal(acc, port.gemmlowp_core(a, b, 4, -6))


@pytest.mark.parametrize("batch,M,N,K,ldd_pad", [(2, 1, 1, 1, 0), (3, 129, 65, 17, 0), (5, 128, 256, 128, 16), (4, 300, 257, 259, 3),
                                                 (7, 31, 593, 23, 0), (2, 257, 130, 1100, 14), (3, 64, 48, 4224, 0), (40, 130, 16, 33, 0)])
def test_batch_in_one_launch(ctx, port, batch, M, N, K, ldd_pad):
    """Products of a batch walked by one launch: tile edges and remainders in every direction, aligned and unaligned rows
    of A, B and dst (canary bytes between and around the products), own and shared B, B that changes with the call."""
    rng = np.random.default_rng(batch * 1000 + K)
    for t, signed in ((np.uint8, False), (np.int8, True)):
        a, b3 = q8_uniform(rng, (batch, M, K), t), q8_uniform(rng, (batch, K, N), t)
        a_off, b_off = (3, -5) if signed else (-128, -120)
        qm, sh = capi.calculate_quantized_multiplier(np.float32(0.5 / (73 * np.sqrt(K))))
        lo, hi = type_range(t)
        bias = rng.integers(-2000, 2001, N).astype(np.int32)
        for b, const in ((b3, False), (b3, True), (b3[0], True)):
            got, kernel = gpu_gemmlowp(ctx, a, b, bias, a_off, b_off, qm, sh, 7, lo, hi, t, b_constant=const, ldd_pad=ldd_pad, runs=2,
                                       temp_workspace=const)
            assert kernel.startswith("tcgen05")
            for i in range(batch):
                want = port.gemmlowp_fused(a[i], b if b.ndim == 2 else b[i], bias, a_off, b_off, [qm], [sh], 7, lo, hi, t)
                assert np.array_equal(got[i], want), (t, const, b.ndim, i)
        acc, _ = gpu_gemmlowp(ctx, a, b3, None, a_off, 0, 0, 0, 0, 0, 0, np.int32, b_constant=False, ldd_pad=ldd_pad)
        assert np.array_equal(acc, port.gemmlowp_core(a, b3, a_off, 0))


def _batch_plan(ctx, batch, M, N, K, ldd_pad=0, **more):
    desc, keep = capi.make_gemm_desc(M, N, K, capi.S8, capi.S8, capi.S8, 5, 0, batch=batch, ldd=N + ldd_pad, b_batch_stride=K * N,
                                     multiplier=2 ** 30, shift=9, min_bound=-128, max_bound=127, **more)
    return capi.GemmPlan(ctx, desc, keep)


def _pair_shape(ctx):
    return 256 * (ctx.sm_count // 4), 512  # a 256 x 256 tile for every pair of SMs (148 SMs: 74 tiles)


def test_batch_routes(ctx):
    """Which batches run in one launch: not those whose products fill the device with a kernel that the batched launch lacks
    (the SM-pair kernel on long K, the channel-major one on ragged rows), and not those told to use such a kernel."""
    M, N = _pair_shape(ctx)
    rows = 256 * ctx.sm_count // 16  # with 1001 columns, eight 128-channel blocks: a channel-major tile for every second SM
    many = 256 * (ctx.sm_count // 4)
    for (m, n, k), launches in (((M, N, 4096), 3), ((M, N, 4080), 1), ((M - 512, N, 4096), 1), ((M + 2048, N, 4096), 1),
                                ((rows + 256, 1001, 96), 3), ((rows + 256, 1008, 96), 1), ((rows - 256, 1001, 96), 1),
                                ((rows + 256, 1001, 528), 1), ((many, 1001, 528), 3), ((many, 1001, 1040), 1), ((many // 2 + 256, 1001, 96), 1),
                                ((384, 384, 128), 1), ((1024, 1024, 1024), 1)):
        plan = _batch_plan(ctx, 3, m, n, k)
        assert plan.launches == launches, (m, n, k)
        plan.close()
    for name, value, launches in (("set_epilogue_warps", 16, 3), ("set_epilogue_warps", 8, 1), ("set_epilogue_warps", 4, 1),
                                  ("set_channel_major", 1, 3), ("set_tile_columns", 64, 1), ("force_simt", True, 3)):
        plan = _batch_plan(ctx, 3, 300, 400, 256)
        getattr(plan, name)(value)
        assert plan.launches == launches, (name, value)
        plan.close()
    plan = _batch_plan(ctx, 3, M, N, 4096)
    plan.allow_pair_kernel(False)
    assert plan.launches == 1
    plan.close()


def test_plan_kernel_of_a_batch(ctx):
    """The kernel a batch's plan names is the one that runs: one CTA per tile in the batched launch, the SM pair only where
    the products go one by one."""
    M, N = _pair_shape(ctx)
    for (m, n, k), kernel in (((M, N, 4096), "tcgen05_2cta"), ((M, N, 2048), "tcgen05"), ((2560, 2560, 1104), "tcgen05"), ((64, 64, 64), "tcgen05")):
        plan = _batch_plan(ctx, 3, m, n, k)
        assert plan.kernel == kernel, (m, n, k)
        plan.close()
    plan = _batch_plan(ctx, 3, M, N, 4096)
    plan.allow_pair_kernel(False)
    assert plan.kernel == "tcgen05"
    plan.close()


@pytest.mark.parametrize("gap,launches", [(0, 1), (16, 1), (5, 2), (8, 2)])
def test_plan_launches_of_a_batch_with_a_gap(ctx, gap, launches):
    """Products of A whose distance is not a multiple of 16 bytes are realigned first: a second launch."""
    plan = _batch_plan(ctx, 3, 40, 64, 32, a_batch_stride=40 * 32 + gap)
    assert plan.launches == launches
    plan.close()


@pytest.mark.parametrize("batch,M,N,K,per_launch,own", [(5, 3000, 33, 5001, 2, True), (5, 3000, 33, 5001, 2, False), (3, 7000, 17, 4999, 1, True),
                                                          (40, 50, 20, 33, 40, True)])
def test_realigned_batches_take_bounded_scratch(ctx, port, batch, M, N, K, per_launch, own):
    """The copies of A that a batch with unaligned rows needs at a time are bounded, whatever the batch: several launches where
    they would be more than 32 MB, the last of them over fewer products; B that changes and B shared by all products."""
    pitch = -(-K // 16) * 16
    plan = _batch_plan(ctx, batch, M, N, K, a_batch_stride=M * K + 16)
    assert plan.temp_bytes == -(-M * per_launch * pitch // 256) * 256 and plan.launches == 2 * -(-batch // per_launch)
    plan.close()
    rng = np.random.default_rng(batch * M + K)
    a, b = q8_uniform(rng, (batch, M, K), np.uint8), q8_uniform(rng, (batch, K, N) if own else (K, N), np.uint8)
    rows = np.unique(np.concatenate([np.arange(40), np.arange(M - 40, M)]))
    for ldd_pad, const in ((0, not own), (3, True)):
        got, _ = gpu_gemmlowp(ctx, a, b, None, -128, -120, 2 ** 30, 12, 3, 0, 255, np.uint8, ldd_pad=ldd_pad, b_constant=const, runs=2,
                              temp_workspace=const)
        for i in range(batch):
            want = port.gemmlowp_fused(a[i][rows], b[i] if own else b, None, -128, -120, [2 ** 30], [12], 3, 0, 255, np.uint8)
            assert np.array_equal(got[i][rows], want), (ldd_pad, const, i)


@pytest.mark.parametrize("batch,M,N,K,ldd_pad,kw", [
    (2, 9472, 512, 4096, 0, {}), (2, 9216, 512, 4096, 0, {}), (2, 2500, 1001, 130, 0, {}), (2, 2100, 1001, 130, 3, {}), (2, 300, 520, 1279, 0, {}),
    (3, 300, 520, 1280, 0, {}), (2, 260, 333, 4095, 0, {}), (2, 260, 333, 4096, 0, {}), (3, 129, 130, 1296, 16, {}), (5, 40, 60, 2000, 0, {}),
    (3, 200, 300, 96, 0, dict(epi_warps=16)), (3, 200, 300, 96, 0, dict(epi_warps=4)), (3, 200, 304, 600, 0, dict(channel_major=1)),
    (3, 200, 304, 1500, 0, dict(epi_warps=8)), (2, 5000, 2304, 64, 0, {})])
def test_batches_on_both_sides_of_the_route_rules(ctx, port, batch, M, N, K, ldd_pad, kw):
    """Products in one launch (four and eight epilogue warps, more than one wave of 256-column tiles) and one by one, against
    the oracle on the first, the last and some rows in between; S32 and F32 too."""
    rng = np.random.default_rng(batch * M + N + K)
    a, b = q8_uniform(rng, (batch, M, K), np.int8), q8_uniform(rng, (batch, K, N), np.int8, -127, 127)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
    shift = rng.integers(8, 14, N).astype(np.int32)
    rows = np.unique(np.concatenate([np.arange(min(M, 40)), rng.integers(0, M, 20), np.arange(max(0, M - 40), M)]))
    got, _ = gpu_gemmlowp(ctx, a, b, None, 5, 0, mult, shift, 3, -128, 127, np.int8, ldd_pad=ldd_pad, **kw)
    raw, _ = gpu_gemmlowp(ctx, a, b, None, 5, 0, 0, 0, 0, 0, 0, np.int32, ldd_pad=4 * (ldd_pad // 4), **kw)
    f, _ = gpu_gemmlowp(ctx, a, b, None, 5, 0, 0, 0, 0, 0, 0, np.float32, dequantize_scale=1.5e-3, b_constant=False, **kw)
    for i in range(batch):
        core = port.gemmlowp_core(a[i][rows], b[i], 5, 0)
        assert np.array_equal(got[i][rows], port.gemmlowp_fused(a[i][rows], b[i], None, 5, 0, mult, shift, 3, -128, 127, np.int8)), i
        assert np.array_equal(raw[i][rows], core), i
        assert np.array_equal(f[i][rows], core.astype(np.float32) * np.float32(1.5e-3)), i


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (5, 63, 19), (129, 65, 130), (40, 4, 127), (33, 1000, 513), (200, 96, 3000)])
def test_operand_preparation(ctx, port, M, N, K):
    """Row sums, realigned rows of A and the K-major copy of B with its column sums, over remainders of every tile edge;
    K ranges one block walks alone and ranges split over blocks."""
    rng = np.random.default_rng(M + K)
    for ta, tb in ((np.uint8, np.uint8), (np.int8, np.int8), (np.uint8, np.int8)):
        a, b = q8_uniform(rng, (M, K), ta), q8_uniform(rng, (K, N), tb)
        for const in (True, False):
            acc, _ = gpu_gemmlowp(ctx, a, b, None, 11, -7, 0, 0, 0, 0, 0, np.int32, b_constant=const, runs=2)
            assert np.array_equal(acc, port.gemmlowp_core(a, b, 11, -7))


@pytest.mark.parametrize("M,K", [(296, 513), (297, 513), (297, 512), (297, 528), (1500, 2064), (20000, 1040)])
@pytest.mark.parametrize("lda_pad", [0, 16, 3])
def test_row_sums_of_many_long_rows(ctx, port, M, K, lda_pad):
    """Row sums alone (aligned rows), with the realigned copy, and a block per row, around the lines between them."""
    import torch
    rng = np.random.default_rng(M + K)
    N, lda = 24, K + lda_pad
    a, b = q8_uniform(rng, (M, lda), np.uint8), q8_uniform(rng, (K, N), np.uint8)
    desc, keep = capi.make_gemm_desc(M, N, K, capi.U8, capi.U8, capi.S32, -128, -120, capi.STAGE_NONE, lda=lda)
    plan = capi.GemmPlan(ctx, desc, keep)
    plan.prepare(torch.from_numpy(b).cuda())
    d_dst = torch.empty((M, N), dtype=torch.int32, device="cuda")
    plan.run(torch.from_numpy(a).cuda(), None, None, d_dst)
    ctx.sync()
    plan.close()
    assert np.array_equal(d_dst.cpu().numpy(), port.gemmlowp_core(np.ascontiguousarray(a[:, :K]), b, -128, -120))


@pytest.mark.parametrize("K,N,ldb", [(1, 1, 1), (3, 2, 5), (130, 63, 63), (257, 65, 67), (513, 130, 131), (900, 429, 429), (131, 64, 66), (70, 7, 7)])
@pytest.mark.parametrize("at", [0, 1, 2, 3])
def test_preparing_b_of_any_alignment(ctx, port, K, N, ldb, at):
    """B whose rows start anywhere: the first and last bytes of the matrix, which no aligned word inside it covers, included."""
    import torch
    rng = np.random.default_rng(K + N + at)
    b, a = q8_uniform(rng, (K, ldb), np.int8), q8_uniform(rng, (5, K), np.int8)
    size = (K - 1) * ldb + N
    d_b = torch.full((size + 64,), 0x7F, dtype=torch.uint8, device="cuda")
    d_b[at:at + size] = torch.from_numpy(b.view(np.uint8).reshape(-1)[:size]).cuda()
    desc, keep = capi.make_gemm_desc(5, N, K, capi.S8, capi.S8, capi.S32, 7, -3, capi.STAGE_NONE, ldb=ldb)
    plan = capi.GemmPlan(ctx, desc, keep)
    plan.prepare(d_b[at:at + size])
    d_dst = torch.empty((5, N), dtype=torch.int32, device="cuda")
    plan.run(torch.from_numpy(a.view(np.uint8)).cuda(), None, None, d_dst)
    ctx.sync()
    plan.close()
    assert np.array_equal(d_dst.cpu().numpy(), port.gemmlowp_core(a, np.ascontiguousarray(b[:, :N]), 7, -3))


@pytest.mark.parametrize("M,N,K", [(1, 64, 2048), (33, 65, 2100), (49, 512, 4608), (97, 31, 16000), (130, 500, 1300), (300, 600, 2000),
                                   (256, 900, 2176), (128, 2112, 2048), (128, 2113, 2048), (128, 8, 2047)])
def test_split_k(ctx, port, M, N, K):
    """Outputs of few tiles, whose K range is shared by clusters of 4 and 8 CTAs: ragged rows, columns and K, K ranges
    that do not divide evenly, every output type and stage encoding, against the oracle and the one-CTA kernel."""
    rng = np.random.default_rng(M + N + K)
    for t, a_off, b_off in ((np.uint8, -128, -120), (np.int8, 5, 0)):
        a, b = q8_uniform(rng, (M, K), t), q8_uniform(rng, (K, N), t)
        lo, hi = type_range(t)
        bias = rng.integers(-2000, 2001, N).astype(np.int32)
        ms = [capi.calculate_quantized_multiplier(np.float32(x / (73 * np.sqrt(K)))) for x in rng.uniform(0.2, 1.0, N)]
        mult, shift = np.array([m for m, _ in ms], np.int32), np.array([s for _, s in ms], np.int32)
        if b_off != 0:
            mult, shift = mult[:1], shift[:1]
        args = (a, b, bias, a_off, b_off, mult if b_off == 0 else int(mult[0]), shift if b_off == 0 else int(shift[0]), 3, lo, hi, t)
        want = port.gemmlowp_fused(a, b, bias, a_off, b_off, mult, shift, 3, lo, hi, t)
        for pad in (0, 5):
            got, _ = gpu_gemmlowp(ctx, *args, ldd_pad=pad, runs=2)
            assert np.array_equal(got, want), (t, pad)
        one, _ = gpu_gemmlowp(ctx, *args, tile_columns=64)
        assert np.array_equal(one, want)
        core = port.gemmlowp_core(a, b, a_off, b_off)
        acc, _ = gpu_gemmlowp(ctx, a, b, None, a_off, b_off, 0, 0, 0, 0, 0, np.int32, ldd_pad=4)
        assert np.array_equal(acc, core)
        init = rng.integers(-1000, 1001, (M, N)).astype(np.int32)
        acc, _ = gpu_gemmlowp(ctx, a, b, None, a_off, b_off, 0, 0, 0, 0, 0, np.int32, accumulate=True, dst_init=init)
        assert np.array_equal(acc, core + init)
        f, _ = gpu_gemmlowp(ctx, a, b, None, a_off, b_off, 0, 0, 0, 0, 0, np.float32, dequantize_scale=0.37e-3)
        assert np.array_equal(f, core.astype(np.float32) * np.float32(0.37e-3))


@pytest.mark.parametrize("M,N,K", [(1, 4, 16), (130, 36, 100), (257, 260, 300), (129, 132, 1500), (1000, 516, 1056), (700, 2052, 144),
                                   (2500, 2052, 1040), (64, 33, 64)])
@pytest.mark.parametrize("ldd_pad", [0, 4])
def test_32_bit_results_through_bulk_stores(ctx, port, M, N, K, ldd_pad):
    """S32 and F32 destinations leave as bulk tensor stores where N and the pitch allow it: every tile width and kernel,
    ragged edges with canary bytes behind each row, against the oracle and the per-lane stores."""
    rng = np.random.default_rng(M + N + K)
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, N), np.int8)
    core = port.gemmlowp_core(a, b, 7, -3)
    for store in (True, False):
        acc, _ = gpu_gemmlowp(ctx, a, b, None, 7, -3, 0, 0, 0, 0, 0, np.int32, ldd_pad=ldd_pad, tma_store=store)
        assert np.array_equal(acc, core), store
        f, _ = gpu_gemmlowp(ctx, a, b, None, 7, -3, 0, 0, 0, 0, 0, np.float32, ldd_pad=ldd_pad, dequantize_scale=1.3e-4, tma_store=store)
        assert np.array_equal(f, core.astype(np.float32) * np.float32(1.3e-4)), store


@pytest.mark.parametrize("M,N,K,ldd_pad", [(300, 9601, 64, 0), (257, 5001, 200, 0), (2400, 1001, 130, 3), (2432, 1024, 1024, 5),
                                           (2400, 1001, 1025, 0), (9700, 129, 16, 2)])
def test_ragged_output_rows(ctx, port, M, N, K, ldd_pad):
    """8-bit rows that are not 16-byte aligned: the channel-major kernel inside its rule, the staged words just outside it
    (K = 1025), canary bytes around every row, per-channel stages of both output types."""
    rng = np.random.default_rng(M + N + K)
    for t, a_off in ((np.uint8, -128), (np.int8, 5)):
        a, b = q8_uniform(rng, (M, K), t), q8_uniform(rng, (K, N), np.int8, -127, 127)
        lo, hi = type_range(t)
        bias = rng.integers(-2000, 2001, N).astype(np.int32)
        mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
        shift = rng.integers(8, 14, N).astype(np.int32)
        got, _ = gpu_gemmlowp(ctx, a, b, bias, a_off, 0, mult, shift, 3, lo, hi, t, ldd_pad=ldd_pad)
        assert np.array_equal(got, port.gemmlowp_fused(a, b, bias, a_off, 0, mult, shift, 3, lo, hi, t)), t


@pytest.mark.parametrize("M,N,ldd_pad", [(2600, 1, 0), (2600, 9, 0), (129, 17, 0), (2600, 24, 8), (2600, 24, 9), (131, 25, 0), (2600, 31, 1), (20000, 63, 0),
                                         (20000, 64, 3), (19000, 65, 0), (300, 72, 0), (300, 152, 1)])
@pytest.mark.parametrize("K", [40, 1300])
def test_few_ragged_columns(ctx, port, M, N, ldd_pad, K):
    """Rows of few unaligned bytes: written byte by byte where they lie close together, as words otherwise, the last short group
    of a wider row, and the channel-major kernel from 65 columns on where there are enough rows."""
    rng = np.random.default_rng(M + N + K)
    a, b = q8_uniform(rng, (M, K), np.uint8), q8_uniform(rng, (K, N), np.int8, -127, 127)
    mult, shift = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32), rng.integers(8, 14, N).astype(np.int32)
    got, _ = gpu_gemmlowp(ctx, a, b, None, -128, 0, mult, shift, 3, 0, 255, np.uint8, ldd_pad=ldd_pad)
    rows = np.unique(np.concatenate([np.arange(100), np.arange(M - 100, M), rng.integers(0, M, 300)]))
    assert np.array_equal(got[rows], port.gemmlowp_fused(a[rows], b, None, -128, 0, mult, shift, 3, 0, 255, np.uint8))


@pytest.mark.parametrize("batch,M,N,K", [(1, 100, 200, 300), (1, 64, 70, 2100), (1, 500, 257, 1000), (3, 40, 96, 640), (16, 384, 384, 128)])
def test_captured_products_with_changing_b(port, batch, M, N, K):
    """A product and a batch whose B (and A) change, recorded into a CUDA graph: operand preparation (with zeroed column sums in
    front of it where K is split over blocks), product and a second product that reads the first one's result, replayed with
    new operands."""
    import torch
    import computelibrary_b200 as cl
    rng = np.random.default_rng(batch * M + N + K)
    stream = torch.cuda.Stream()
    ctx = cl.Context(0, stream.cuda_stream)
    mult, shift = capi.calculate_quantized_multiplier(np.float32(0.5 / (73 * np.sqrt(K))))
    mult2, shift2 = capi.calculate_quantized_multiplier(np.float32(0.5 / (73 * np.sqrt(N))))

    def plan_for(m, n, k, mu, sh):
        desc, keep = capi.make_gemm_desc(m, n, k, capi.U8, capi.U8, capi.U8, -128, -120, batch=batch, b_batch_stride=k * n if batch > 1 else 0,
                                         multiplier=mu, shift=sh, offset=100, min_bound=0, max_bound=255, b_constant=False)
        return capi.GemmPlan(ctx, desc, keep)
    first, second = plan_for(M, N, K, mult, shift), plan_for(M, 48, N, mult2, shift2)
    shapes = ((batch, M, K), (batch, K, N), (batch, N, 48))
    with torch.cuda.stream(stream):
        d_a, d_b, d_c = (torch.empty(s, dtype=torch.uint8, device="cuda") for s in shapes)
        d_mid, d_out = (torch.empty((batch, M, n), dtype=torch.uint8, device="cuda") for n in (N, 48))

        def step():
            first.run(d_a, d_b, None, d_mid)
            second.run(d_mid, d_c, None, d_out)
        step()
    ctx.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        step()
    for _ in range(3):
        a, b, c = (q8_uniform(rng, s, np.uint8) for s in shapes)
        with torch.cuda.stream(stream):
            for d, h in ((d_a, a), (d_b, b), (d_c, c)):
                d.copy_(torch.from_numpy(h))
            graph.replay()
        ctx.sync()
        for i in range(batch):
            mid = port.gemmlowp_fused(a[i], b[i], None, -128, -120, [mult], [shift], 100, 0, 255, np.uint8)
            assert np.array_equal(d_mid[i].cpu().numpy(), mid), i
            assert np.array_equal(d_out[i].cpu().numpy(), port.gemmlowp_fused(mid, c[i], None, -128, -120, [mult2], [shift2], 100, 0, 255, np.uint8)), i
    del graph
    first.close()
    second.close()
    ctx.close()


def test_run_twice_and_variable_b(ctx, port):
    """MultipleExecution (GEMMLowp.cpp:211-297): same plan, same output; B re-laid out per run when it is
    not constant (reshape_b_only_on_first_run = false)."""
    rng = np.random.default_rng(6)
    a, b = q8_uniform(rng, (200, 160), np.uint8), q8_uniform(rng, (160, 300), np.uint8)
    qm, sh = capi.calculate_quantized_multiplier(np.float32(0.0004))
    want = port.gemmlowp_fused(a, b, None, -100, -90, [qm], [sh], 5, 0, 255, np.uint8)
    for const in (True, False):
        got, _ = gpu_gemmlowp(ctx, a, b, None, -100, -90, qm, sh, 5, 0, 255, np.uint8, b_constant=const, runs=3)
        assert np.array_equal(got, want)


def test_update_quantization_parameters(ctx, port):
    import torch
    rng = np.random.default_rng(8)
    M, N, K = 96, 80, 64
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, N), np.int8)
    d1, k1 = capi.make_gemm_desc(M, N, K, capi.S8, capi.S8, capi.S8, 2, 0, multiplier=2 ** 30, shift=6, offset=0,
                                 min_bound=-128, max_bound=127)
    plan = capi.GemmPlan(ctx, d1, k1)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    dd = torch.empty((M, N), dtype=torch.int8, device="cuda")
    plan.prepare(db)
    plan.run(da, None, None, dd)
    ctx.sync()
    assert np.array_equal(dd.cpu().numpy(), port.gemmlowp_fused(a, b, None, 2, 0, [2 ** 30], [6], 0, -128, 127, np.int8))
    d2, k2 = capi.make_gemm_desc(M, N, K, capi.S8, capi.S8, capi.S8, -9, 4, multiplier=1518500250, shift=5, offset=-4,
                                 min_bound=-100, max_bound=90)
    plan.update_quantization(d2, k2)
    plan.run(da, None, None, dd)
    ctx.sync()
    assert np.array_equal(dd.cpu().numpy(),
                          port.gemmlowp_fused(a, b, None, -9, 4, [1518500250], [5], -4, -100, 90, np.int8))
    plan.close()


@pytest.mark.parametrize("shape,b_dtype,b_off", [((256, 192, 128), np.int8, 0), ((2600, 320, 192), np.int8, 0),
                                                 ((4099, 136, 80), np.uint8, -7)])
def test_run_host_end_to_end(ctx, port, shape, b_dtype, b_off):
    """The host-buffer entry point: pinned buffers in, pinned buffers out; from 2048 rows on the call pipelines
    row blocks (copy in / multiply / copy out) over three streams, with ragged last blocks and row sums."""
    import ctypes as C
    rng = np.random.default_rng(10)
    M, N, K = shape
    a, b = q8_uniform(rng, (M, K), np.uint8), q8_uniform(rng, (K, N), b_dtype)
    bias = rng.integers(-1000, 1000, N).astype(np.int32)
    import torch
    desc, keep = capi.make_gemm_desc(M, N, K, capi.U8, capi.S8 if b_dtype == np.int8 else capi.U8, capi.U8, -128, b_off,
                                     multiplier=2 ** 30, shift=9, offset=3, min_bound=0, max_bound=255, has_bias=True)
    plan = capi.GemmPlan(ctx, desc, keep)
    plan.prepare(torch.from_numpy(b.view(np.uint8)).cuda())
    h_a, h_d, h_b = ctx.host_alloc(M * K), ctx.host_alloc(M * N), ctx.host_alloc(N * 4)
    C.memmove(h_a, a.ctypes.data, M * K)
    C.memmove(h_b, bias.ctypes.data, N * 4)
    want = port.gemmlowp_fused(a, b, bias, -128, b_off, [2 ** 30], [9], 3, 0, 255, np.uint8)
    for _ in range(2):
        C.memset(h_d, 0xEE, M * N)
        plan.run_host(h_a, h_b, h_d)
        got = np.ctypeslib.as_array((C.c_uint8 * (M * N)).from_address(h_d)).reshape(M, N).copy()
        assert np.array_equal(got, want)
    for p in (h_a, h_d, h_b):
        ctx.host_free(p)
    plan.close()


def test_config2_full_size_properties(ctx, port):
    """4096^3 (configuration 2 of the benchmark): exact on a row sample against the oracle, tensor-core and generic kernels
    agree everywhere, and the result is invariant under a row permutation of A (rows are independent)."""
    c = config2()
    mult, shift = f32_mults(port, c["i_scale"], c["w_scales"], c["o_scale"])
    out, kern = gpu_gemmlowp(ctx, c["a"], c["b"], c["bias"], c["a_off"], 0, mult, shift, 0, -128, 127, np.int8)
    assert kern == "tcgen05_2cta"
    rows = np.r_[0:64, 2000:2064, 4032:4096]
    want = port.gemmlowp_fused(c["a"][rows], c["b"], c["bias"], c["a_off"], 0, mult, shift, 0, -128, 127, np.int8)
    assert np.array_equal(out[rows], want)
    ref2, _ = gpu_gemmlowp(ctx, c["a"], c["b"], c["bias"], c["a_off"], 0, mult, shift, 0, -128, 127, np.int8,
                           force_simt=True)
    assert np.array_equal(out, ref2)
    one_cta, kern1 = gpu_gemmlowp(ctx, c["a"], c["b"], c["bias"], c["a_off"], 0, mult, shift, 0, -128, 127, np.int8,
                                  pair=False)
    assert kern1 == "tcgen05" and np.array_equal(out, one_cta)
    perm = np.random.default_rng(0).permutation(4096)
    outp, _ = gpu_gemmlowp(ctx, c["a"][perm], c["b"], c["bias"], c["a_off"], 0, mult, shift, 0, -128, 127, np.int8)
    assert np.array_equal(outp, out[perm])
    assert 0.05 < np.mean(np.abs(out.astype(np.int32)) == 127 + (out < 0)) < 0.999  # not all saturated


def test_config5_column_shard_property(ctx, port):
    """Config 5 at reduced M: a column shard of B gives exactly the same columns as the full GEMM (what the
    N-sharded multi-GPU run relies on), and a row sample matches the oracle."""
    c = config5(M=512)
    mult, shift = f32_mults(port, c["i_scale"], c["w_scales"], c["o_scale"])
    full, _ = gpu_gemmlowp(ctx, c["a"], c["b"], None, 0, 0, mult, shift, 0, -128, 127, np.int8)
    want = port.gemmlowp_fused(c["a"][:48], c["b"], None, 0, 0, mult, shift, 0, -128, 127, np.int8)
    assert np.array_equal(full[:48], want)
    n0, n1 = 1792 * 3, 1792 * 4
    shard, _ = gpu_gemmlowp(ctx, c["a"], np.ascontiguousarray(c["b"][:, n0:n1]), None, 0, 0, mult[n0:n1],
                            shift[n0:n1], 0, -128, 127, np.int8)
    assert np.array_equal(shard, full[:, n0:n1])


def test_run_multi_destinations(ctx, port):
    """The push all-gather epilogue: one launch writes the same column block into several [M, N_total] matrices
    (here three buffers on one GPU; across GPUs the extra pointers are the peers' buffers)."""
    import torch
    rng = np.random.default_rng(21)
    M, K, n_local, n_total, n0 = 300, 256, 512, 1536, 512
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, n_local), np.int8, -127, 127)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, n_local).astype(np.int32)
    shift = rng.integers(5, 10, n_local).astype(np.int32)
    desc, keep = capi.make_gemm_desc(M, n_local, K, capi.S8, capi.S8, capi.S8, 0, 0, multipliers=mult, shifts=shift,
                                     min_bound=-128, max_bound=127, ldd=n_total)
    plan = capi.GemmPlan(ctx, desc, keep)
    plan.prepare(torch.from_numpy(b.view(np.uint8)).cuda())
    d_a = torch.from_numpy(a.view(np.uint8)).cuda()
    bufs = [torch.full((M, n_total), 0x11, dtype=torch.uint8, device="cuda") for _ in range(3)]
    plan.run_multi(d_a, None, [t.data_ptr() + n0 for t in bufs])
    ctx.sync()
    want = port.gemmlowp_fused(a, b, None, 0, 0, mult, shift, 0, -128, 127, np.int8)
    for t in bufs:
        h = t.cpu().numpy()
        assert np.array_equal(h[:, n0:n0 + n_local].view(np.int8), want)
        assert (h[:, :n0] == 0x11).all() and (h[:, n0 + n_local:] == 0x11).all()
    plan.close()


@pytest.mark.parametrize("epi_warps", [4, 8, 16])
@pytest.mark.parametrize("shape", [(300, 256, 64), (257, 96, 128), (130, 40, 2048), (515, 520, 320), (128, 64, 16)])
def test_epilogue_builds_and_stage_encodings(ctx, port, shape, epi_warps):
    """Both builds of the tensor-core kernels (four / eight epilogue warps) on all three encodings of the output
    stage: shifts >= 2 with non-negative multipliers (one wide multiply-add per element), shifts 0 and 1 (two
    half multiplies), and left shifts / INT32_MIN multipliers (the reference expression as written)."""
    M, N, K = shape
    rng = np.random.default_rng(M + N + K + epi_warps)
    a, b = q8_uniform(rng, (M, K), np.uint8), q8_uniform(rng, (K, N), np.int8, -127, 127)
    bias = rng.integers(-20000, 20001, N).astype(np.int32)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
    for lo_shift, hi_shift, label in [(2, 14, "wide"), (0, 6, "fast"), (-2, 5, "generic")]:
        shift = rng.integers(lo_shift, hi_shift, N).astype(np.int32)
        shift[0], shift[-1] = lo_shift, hi_shift - 1
        want = port.gemmlowp_fused(a, b, bias, -7, 0, mult, shift, 3, 0, 255, np.uint8)
        # channel-major: 8-byte aligned rows take the shared-memory byte transpose, a pitch of N + 5 the byte stores
        for pair, cm, pad in ((True, -1, 0), (False, -1, 0), (False, 1, 0), (False, 1, 5), (False, 1, 8)):
            got, kern = gpu_gemmlowp(ctx, a, b, bias, -7, 0, mult, shift, 3, 0, 255, np.uint8, pair=pair,
                                     epi_warps=epi_warps, channel_major=cm, ldd_pad=pad)
            assert kern.startswith("tcgen05")
            assert np.array_equal(got, want), (label, pair, cm, pad, np.argwhere(got != want)[:4])
        # these outputs have fewer tiles than the device has SMs, so the library narrows the tiles by itself; the
        # forced widths cover every tile variant of the build (256 is the only one of the sixteen-warp build)
        for cols in (256, 128, 64):
            got, kern = gpu_gemmlowp(ctx, a, b, bias, -7, 0, mult, shift, 3, 0, 255, np.uint8, epi_warps=epi_warps,
                                     channel_major=-1, tile_columns=cols)
            assert kern.startswith("tcgen05")
            assert np.array_equal(got, want), (label, cols, np.argwhere(got != want)[:4])
    # per-tensor wide encoding with a signed output and a lower bound above the type minimum
    a8 = q8_uniform(rng, (M, K), np.int8)
    got, _ = gpu_gemmlowp(ctx, a8, b, bias, 5, 0, 1759218688, 13, -3, -100, 90, np.int8, epi_warps=epi_warps)
    assert np.array_equal(got, port.gemmlowp_fused(a8, b, bias, 5, 0, [1759218688], [13], -3, -100, 90, np.int8))
    # raw int32 accumulators with the offset terms, row-major and channel-major kernels
    for cm in (-1, 1):
        got, _ = gpu_gemmlowp(ctx, a, b, None, -7, 0, 0, 0, 0, 0, 0, np.int32, epi_warps=epi_warps, channel_major=cm)
        assert np.array_equal(got, port.gemmlowp_core(a, b, -7, 0)), cm
    # asymmetric weights (row-sum term present): never the wide encoding
    bu = q8_uniform(rng, (K, N), np.uint8)
    got, _ = gpu_gemmlowp(ctx, a, bu, bias, -7, -9, 1099511552, 8, 10, 0, 255, np.uint8, epi_warps=epi_warps)
    assert np.array_equal(got, port.gemmlowp_fused(a, bu, bias, -7, -9, [1099511552], [8], 10, 0, 255, np.uint8))


@pytest.mark.parametrize("M,N,K,pad,n", [(300, 520, 96, 8, 3), (300, 520, 96, 0, 8), (2400, 1024, 64, 0, 2), (129, 333, 200, 0, 4), (257, 96, 1300, 0, 8),
                                         (4736, 512, 1040, 16, 3), (70, 17, 640, 0, 5)])
@pytest.mark.parametrize("epi_warps", [0, 4, 8, 16])
def test_run_multi_every_store_path(ctx, port, M, N, K, pad, n, epi_warps):
    """The push to several destinations on every kernel that writes them: whole and ragged pieces, unaligned and short rows, wide
    and narrow tiles, the SM pair; canary bytes between and behind the rows of each destination; 32-bit results as well."""
    import torch
    rng = np.random.default_rng(M + N + K + n)
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, N), np.int8, -127, 127)
    mult, shift = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32), rng.integers(8, 14, N).astype(np.int32)
    rows = np.unique(np.concatenate([np.arange(min(M, 70)), np.arange(max(0, M - 70), M)]))
    d_a, d_b = torch.from_numpy(a.view(np.uint8)).cuda(), torch.from_numpy(b.view(np.uint8)).cuda()
    for out, want in ((capi.S8, port.gemmlowp_fused(a[rows], b, None, 5, 0, mult, shift, 3, -128, 127, np.int8)),
                      (capi.S32, port.gemmlowp_core(a[rows], b, 5, 0))):
        size = want.dtype.itemsize
        ldd = N * size + 4 * pad
        stage = dict(stage=capi.STAGE_NONE) if out == capi.S32 else dict(multipliers=mult, shifts=shift, offset=3, min_bound=-128, max_bound=127)
        desc, keep = capi.make_gemm_desc(M, N, K, capi.S8, capi.S8, out, 5, 0, ldd=ldd, **stage)
        plan = capi.GemmPlan(ctx, desc, keep)
        plan.set_epilogue_warps(epi_warps)
        plan.prepare(d_b)
        dsts = [torch.full((M * ldd + 64,), 0xA5, dtype=torch.uint8, device="cuda") for _ in range(n)]
        plan.run_multi(d_a, None, dsts)
        ctx.sync()
        for d in dsts:
            got = d.cpu().numpy()
            body = got[:M * ldd].reshape(M, ldd)
            assert np.array_equal(np.ascontiguousarray(body[rows][:, :N * size]).view(want.dtype), want), out
            assert (body[:, N * size:] == 0xA5).all() and (got[M * ldd:] == 0xA5).all(), out
        plan.close()


def test_run_multi_destinations_eight_epilogue_warps(ctx, port):
    """The staged multi-destination store of the eight-warp build (64-byte row segments), ragged N and M."""
    import torch
    rng = np.random.default_rng(22)
    M, K, n_local, n_total, n0 = 301, 128, 400, 1200, 400
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, n_local), np.int8, -127, 127)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, n_local).astype(np.int32)
    shift = rng.integers(5, 10, n_local).astype(np.int32)
    want = port.gemmlowp_fused(a, b, None, 0, 0, mult, shift, 0, -128, 127, np.int8)
    for warps in (4, 8, 16):
        desc, keep = capi.make_gemm_desc(M, n_local, K, capi.S8, capi.S8, capi.S8, 0, 0, multipliers=mult, shifts=shift,
                                         min_bound=-128, max_bound=127, ldd=n_total)
        plan = capi.GemmPlan(ctx, desc, keep)
        plan.set_epilogue_warps(warps)
        plan.prepare(torch.from_numpy(b.view(np.uint8)).cuda())
        d_a = torch.from_numpy(a.view(np.uint8)).cuda()
        bufs = [torch.full((M, n_total), 0x11, dtype=torch.uint8, device="cuda") for _ in range(2)]
        plan.run_multi(d_a, None, [t.data_ptr() + n0 for t in bufs])
        ctx.sync()
        for t in bufs:
            h = t.cpu().numpy()
            assert np.array_equal(h[:, n0:n0 + n_local].view(np.int8), want), warps
            assert (h[:, :n0] == 0x11).all() and (h[:, n0 + n_local:] == 0x11).all()
        plan.close()


@pytest.mark.parametrize("shape", [(2304, 2304, 1152), (2290, 2200, 1136), (1024, 5000, 1040)])
def test_pair_kernel_tail_split(ctx, port, shape):
    """SM-pair kernel with a short last wave (81, 81 and 80 tiles of 256 x 256 on 74 SM pairs): the tail tiles run
    as two 256 x 128 halves.  Same bytes as the oracle and as the unsplit kernel, ragged edges included."""
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, N), np.int8, -127, 127)
    bias = rng.integers(-20000, 20001, N).astype(np.int32)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
    shift = rng.integers(6, 12, N).astype(np.int32)
    want = port.gemmlowp_fused(a, b, bias, 5, 0, mult, shift, -3, -128, 127, np.int8)
    outs = []
    for split in (True, False):
        import torch
        desc, keep = capi.make_gemm_desc(M, N, K, capi.S8, capi.S8, capi.S8, 5, 0, multipliers=mult, shifts=shift,
                                         offset=-3, min_bound=-128, max_bound=127, has_bias=True)
        plan = capi.GemmPlan(ctx, desc, keep)
        plan.set_tail_split(split)
        assert plan.kernel == "tcgen05_2cta"
        plan.prepare(torch.from_numpy(b.view(np.uint8)).cuda())
        d_dst = torch.full((M, N), 0x55, dtype=torch.uint8, device="cuda")
        plan.run(torch.from_numpy(a.view(np.uint8)).cuda(), None, torch.from_numpy(bias).cuda(), d_dst)
        ctx.sync()
        outs.append(d_dst.cpu().numpy().view(np.int8))
        plan.close()
    assert np.array_equal(outs[0], want), np.argwhere(outs[0] != want)[:5]
    assert np.array_equal(outs[1], want)


@pytest.mark.parametrize("force_simt", [False, True])
def test_fused_quantize_down_stage_golden(ctx, port, gemm_golden, force_simt):
    """NEGEMMLowpMatrixMultiplyCore with a fused QUANTIZE_DOWN (integer multiply) stage against the reference
    fixtures: per-channel and per-tensor, tensor-core (where TMA can address the operands) and generic kernels."""
    for g in golden_gemm_cases():
        im, ish, ioff, ilo, ihi = golden_int_stage(g)
        od = g["out_dtype"]
        got, _ = gpu_gemmlowp(ctx, g["a"], g["b"], g["bias"], g["a_off"], 0, im, ish, ioff, ilo, ihi, od,
                              force_simt=force_simt, integer_stage=True)
        assert np.array_equal(got, gemm_golden[g["key"] + "_int_pc"]), g["key"]
        got, _ = gpu_gemmlowp(ctx, g["a"], g["b"], g["bias"], g["a_off"], g["b_off"], int(im[0]), int(ish[0]), ioff, ilo,
                              ihi, od, force_simt=force_simt, integer_stage=True)
        assert np.array_equal(got, gemm_golden[g["key"] + "_int_pt"]), g["key"]


def test_fused_quantize_down_stage_tensor_core_shapes(ctx, port):
    rng = np.random.default_rng(91)
    for (M, N, K) in [(300, 256, 64), (515, 520, 1088), (130, 40, 2048)]:
        a, b = q8_uniform(rng, (M, K), np.uint8), q8_uniform(rng, (K, N), np.int8, -127, 127)
        bias = rng.integers(-20000, 20001, N).astype(np.int32)
        mult = rng.integers(1, 60, N).astype(np.int32)
        shift = rng.integers(8, 16, N).astype(np.int32)
        want = port.gemmlowp_fused_int(a, b, bias, -9, 0, mult, shift, 4000, 3, 250, np.uint8)
        got, kern = gpu_gemmlowp(ctx, a, b, bias, -9, 0, mult, shift, 4000, 3, 250, np.uint8, integer_stage=True)
        assert kern.startswith("tcgen05") and np.array_equal(got, want), (M, N, K)
        want = port.gemmlowp_fused_int(a, b, None, -9, 0, mult, shift, 4000, 0, 0, np.uint8)   # equal bounds: type range
        got, _ = gpu_gemmlowp(ctx, a, b, None, -9, 0, mult, shift, 4000, 0, 0, np.uint8, integer_stage=True)
        assert np.array_equal(got, want), (M, N, K)


@pytest.mark.parametrize("epi_warps", [4, 8, 16])
@pytest.mark.parametrize("shape", [(38477, 256, 64), (20000, 520, 96), (37900, 300, 496)])
def test_paired_drain(ctx, port, shape, epi_warps):
    """More 128 x 256 tiles than SMs, so a CTA owns several: consecutive tiles of one column block are drained from
    the two accumulator buffers together (one term read for two elements), with single tiles left over where the
    column block changes or the count is odd.  Same bytes as the oracle and as the unpaired epilogue."""
    M, N, K = shape
    rng = np.random.default_rng(M + N + K + epi_warps)
    a, b = q8_uniform(rng, (M, K), np.uint8), q8_uniform(rng, (K, N), np.int8, -127, 127)
    bias = rng.integers(-20000, 20001, N).astype(np.int32)
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
    shift = rng.integers(2, 12, N).astype(np.int32)
    want = port.gemmlowp_fused(a, b, bias, -7, 0, mult, shift, 3, 0, 255, np.uint8)
    for paired in (True, False):
        got, kern = gpu_gemmlowp(ctx, a, b, bias, -7, 0, mult, shift, 3, 0, 255, np.uint8, pair=False,
                                 epi_warps=epi_warps, channel_major=-1, paired_drain=paired)
        assert kern == "tcgen05"
        assert np.array_equal(got, want), (paired, np.argwhere(got != want)[:4])


# Shapes of tests/datasets/SmallGEMMLowpDataset.h:43-52 and LargeGEMMLowpDataset.h:43-52 as (M, N, K, a_offset, b_offset)
REFERENCE_DATASET_SHAPES = [(13, 33, 21, 0, 0), (13, 33, 52, 0, 4), (27, 23, 31, 18, 23), (72, 17, 32, -9, 1),
                            (1, 33, 21, 0, 0), (13, 1, 21, 5, 13), (973, 221, 1021, 10, 2), (1123, 213, 941, -3, -2),
                            (429, 71, 1021, 1, -1), (1023, 171, 1, 1, 3)]


@pytest.mark.parametrize("M,N,K,ao,bo", REFERENCE_DATASET_SHAPES)
def test_reference_dataset_shapes_run_on_the_tensor_cores(ctx, port, M, N, K, ao, bo):
    """Every shape of the reference's Small / Large GEMMLowp datasets -- K and row pitches that are no multiples of 16
    among them -- runs on the tcgen05 kernel (through a 16-byte-pitch copy of A where needed) and is exact."""
    rng = np.random.default_rng(M * 7 + K)
    a, b = q8_uniform(rng, (M, K), np.uint8), q8_uniform(rng, (K, N), np.uint8)
    got, kern = gpu_gemmlowp(ctx, a, b, None, ao, bo, 0, 0, 0, 0, 0, np.int32)
    assert kern.startswith("tcgen05"), kern
    assert np.array_equal(got, port.gemmlowp_core(a, b, ao, bo))
    bias = rng.integers(-3000, 3001, N).astype(np.int32)
    mult, shift = 1518500250, int(np.ceil(np.log2(max(K, 2) * 255 * 255 / 200)))
    got, kern = gpu_gemmlowp(ctx, a, b, bias, ao, bo, mult, shift, 7, 0, 255, np.uint8, temp_workspace=True)
    assert kern.startswith("tcgen05"), kern
    assert np.array_equal(got, port.gemmlowp_fused(a, b, bias, ao, bo, [mult], [shift], 7, 0, 255, np.uint8))


@pytest.mark.parametrize("M,N,K", [(70, 130, 221), (256, 512, 1040), (300, 64, 96)])
@pytest.mark.parametrize("force_simt", [False, True])
def test_accumulate_and_dequantized_output(ctx, port, M, N, K, force_simt):
    """GEMMInfo::accumulate (dst += A * B, S32) and the s8 x s8 -> F32 rows of the type table: float(int32) * scale with
    one rounding each, identical to the reference's dequantization of the S32 result bit for bit."""
    rng = np.random.default_rng(M + N + K)
    a, b = q8_uniform(rng, (M, K), np.int8), q8_uniform(rng, (K, N), np.int8)
    acc = port.gemmlowp_core(a, b, 3, -4)
    start = rng.integers(-2 ** 20, 2 ** 20, (M, N)).astype(np.int32)
    got, _ = gpu_gemmlowp(ctx, a, b, None, 3, -4, 0, 0, 0, 0, 0, np.int32, accumulate=True, dst_init=start, runs=2,
                          force_simt=force_simt, ldd_pad=4)
    assert np.array_equal(got, start + 2 * acc)
    scale = float(np.float32(1 / 255) * np.float32(5 / 255))
    got, _ = gpu_gemmlowp(ctx, a, b, None, 3, -4, 0, 0, 0, 0, 0, np.float32, dequantize_scale=scale, force_simt=force_simt)
    want = port.dequantize_s32(acc, scale)
    assert got.dtype == np.float32 and np.array_equal(got, want)
    prev = rng.uniform(-100, 100, (M, N)).astype(np.float32)
    got, _ = gpu_gemmlowp(ctx, a, b, None, 3, -4, 0, 0, 0, 0, 0, np.float32, dequantize_scale=scale, accumulate=True,
                          dst_init=prev, force_simt=force_simt)
    assert np.array_equal(got, port.dequantize_s32(acc, scale, prev))


@pytest.mark.parametrize("M,N,K", [(129, 33, 40), (257, 260, 600), (300, 1001, 1100), (95, 96, 2100), (1000, 31, 64), (31, 512, 1040)])
@pytest.mark.parametrize("ldd_pad", [0, 3, 4])
def test_accumulation_into_any_rows(ctx, port, M, N, K, ldd_pad):
    """dst += result into rows of every alignment, with whole and partial chunks of 32 rows and 32 columns, one product and a
    batch, four and eight epilogue warps and a cluster per tile (K = 2100)."""
    rng = np.random.default_rng(M + N + K)
    a, b = q8_uniform(rng, (2, M, K), np.int8), q8_uniform(rng, (2, K, N), np.int8)
    cores = np.stack([port.gemmlowp_core(a[i], b[i], 7, -3) for i in range(2)])
    init = rng.integers(-2 ** 20, 2 ** 20, (2, M, N)).astype(np.int32)
    for n in (1, 2):
        ops = (a[0], b[0]) if n == 1 else (a, b)
        core, start = (cores[0], init[0]) if n == 1 else (cores, init)
        got, _ = gpu_gemmlowp(ctx, *ops, None, 7, -3, 0, 0, 0, 0, 0, np.int32, ldd_pad=ldd_pad, accumulate=True, dst_init=start, runs=2)
        assert np.array_equal(got, start + 2 * core), n
        prev = start.astype(np.float32) * np.float32(0.25)
        got, _ = gpu_gemmlowp(ctx, *ops, None, 7, -3, 0, 0, 0, 0, 0, np.float32, ldd_pad=ldd_pad, accumulate=True, dst_init=prev, dequantize_scale=0.125)
        assert np.array_equal(got, prev + core.astype(np.float32) * np.float32(0.125)), n


@pytest.mark.parametrize("M,N,K", [(4096, 4096, 4096), (2048, 2048, 1024), (2000, 2001, 1024)])
def test_accumulation_is_no_chain_of_round_trips(ctx, M, N, K):
    """Adding into dst reads its old values many rows at a time: it costs a small multiple of overwriting dst (1.2 - 1.8 measured),
    not the 5 - 8 of a load that waits for the store of the row before it."""
    import torch
    a, b = (torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda") for n in (M * K, K * N))
    dst = torch.zeros(M * N, dtype=torch.int32, device="cuda")
    best = {}
    for accumulate in (False, True):
        desc, keep = capi.make_gemm_desc(M, N, K, capi.S8, capi.S8, capi.S32, 5, 0, capi.STAGE_NONE, accumulate=accumulate)
        plan = capi.GemmPlan(ctx, desc, keep)
        plan.prepare(b)
        times = []
        for _ in range(8):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(5):
                plan.run(a, None, None, dst)
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        best[accumulate] = min(times)
        plan.close()
    assert best[True] < 3 * best[False], best


def test_validate_rules_of_the_raw_outputs():
    d, keep = capi.make_gemm_desc(8, 8, 8, capi.S8, capi.S8, capi.F32, stage=capi.STAGE_NONE)
    assert capi.gemm_validate(d)[0] == 6            # an F32 output needs a scale
    d, keep = capi.make_gemm_desc(8, 8, 8, capi.S8, capi.S8, capi.F32, stage=capi.STAGE_NONE, dequantize_scale=0.1)
    assert capi.gemm_validate(d)[0] == 0
    d, keep = capi.make_gemm_desc(8, 8, 8, capi.S8, capi.S8, capi.S8, multiplier=2 ** 30, shift=1, accumulate=True)
    assert capi.gemm_validate(d)[0] == 6            # accumulation only without an output stage


@pytest.mark.parametrize("out_dtype,offset", [(np.uint8, 0), (np.uint8, 7), (np.int8, 0), (np.int8, -11)])
@pytest.mark.parametrize("M,N,K,epi", [(300, 256, 64, 0), (257, 512, 192, 0), (520, 320, 2048, 0), (130, 64, 96, 8), (1000, 256, 512, 1)])
def test_saturating_pack_encoding(ctx, port, out_dtype, offset, M, N, K, epi):
    """Whole-type-range clamps run on the saturating-pack encoding of the output stage (offset folded into the column
    constant, cvt.pack.sat as the clamp): identical to the explicit encoding and to the oracle, for results far
    outside the type range on both sides, shifts up to the limit of the encoding and beyond it."""
    rng = np.random.default_rng(M + N + K + offset)
    a_dt = np.uint8 if out_dtype == np.uint8 else np.int8
    a, b = q8_uniform(rng, (M, K), a_dt), q8_uniform(rng, (K, N), np.int8, -127, 127)
    bias = rng.integers(-400000, 400001, N).astype(np.int32)   # drives many results beyond both ends of the range
    mult = rng.integers(2 ** 30, 2 ** 31 - 1, N).astype(np.int32)
    lo, hi = type_range(out_dtype)
    for max_shift in (12, 22, 24):
        shift = rng.integers(2, max_shift + 1, N).astype(np.int32)
        shift[0] = max_shift
        want = port.gemmlowp_fused(a, b, bias, 3, 0, mult, shift, offset, lo, hi, out_dtype)
        kw = dict(channel_major=1) if epi == 1 else dict(epi_warps=epi)
        got, _ = gpu_gemmlowp(ctx, a, b, bias, 3, 0, mult, shift, offset, lo, hi, out_dtype, **kw)
        ref, _ = gpu_gemmlowp(ctx, a, b, bias, 3, 0, mult, shift, offset, lo, hi, out_dtype, saturating_pack=False, **kw)
        assert np.array_equal(got, want) and np.array_equal(ref, want), max_shift


@pytest.mark.parametrize("shape", [(300, 200, 64), (300, 208, 64), (700, 520, 64), (1000, 96, 256), (2049, 333, 1536), (40000, 256, 64),
                                   (20000, 64, 128)])
def test_bulk_tensor_stores_against_per_lane_stores(ctx, port, shape):
    """The epilogue's two ways of writing the output -- a warp's rows as one bulk tensor store from shared memory, or
    one store per lane -- on ragged M and N, narrow and wide tiles, short and long K: both against the oracle (a row
    sample for the large cases) and against each other, with a canary pitch that makes the destination rows 16-byte
    aligned (bulk stores possible) or not (the plan must fall back to per-lane stores by itself)."""
    M, N, K = shape
    r = np.random.default_rng(M + N + K)
    a, b = q8_uniform(r, (M, K), np.uint8), q8_uniform(r, (K, N), np.int8, -127, 127)
    bias = r.integers(-4000, 4000, N).astype(np.int32)
    ws = np.exp(r.uniform(np.log(1e-3), np.log(1e-2), N)).astype(np.float32)
    mult, shift = f32_mults(port, 0.05, ws, 0.05 * max(1, K // 64))
    rows = np.unique(np.concatenate([np.arange(0, min(M, 300)), np.arange(max(0, M - 300), M)]))
    want = port.gemmlowp_fused(a[rows], b, bias, -3, 0, mult, shift, 5, 0, 255, np.uint8)
    outs = []
    for tma, pad in ((True, 0), (False, 0), (True, 16 - N % 16 if N % 16 else 16), (True, 3)):
        out, _ = gpu_gemmlowp(ctx, a, b, bias, -3, 0, mult, shift, 5, 0, 255, np.uint8, ldd_pad=pad, tma_store=tma)
        assert np.array_equal(out[rows], want), (tma, pad)
        outs.append(out)
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])


@pytest.mark.parametrize("widths", [(256, 256, 256), (64, 320, 128), (1024, 64, 512)])
def test_chained_launches_with_and_without_dependent_launch(ctx, port, widths):
    """A chain of three GEMMs, each reading what the one before it wrote, launched back to back twenty times over the
    same buffers (so that a kernel also overwrites what its predecessor is still reading unless it waits for it): with
    programmatic stream serialization (the default outside graph capture) and with plain stream order the chain ends
    in the same bytes, equal to the oracle's."""
    import torch
    M, K0 = 3000, 128
    r = np.random.default_rng(sum(widths))
    a = q8_uniform(r, (M, K0), np.uint8)
    dims = (K0,) + widths
    layers, want = [], a
    for k, n in zip(dims[:-1], dims[1:]):
        b = q8_uniform(r, (k, n), np.int8, -127, 127)
        bias = r.integers(-3000, 3000, n).astype(np.int32)
        ws = np.exp(r.uniform(np.log(1e-3), np.log(4e-3), n)).astype(np.float32)
        mult, shift = f32_mults(port, 0.05, ws, 0.05 * max(1, k // 128))
        want = port.gemmlowp_fused(want, b, bias, -2, 0, mult, shift, 4, 0, 255, np.uint8)
        layers.append((k, n, b, bias, mult, shift))
    results = {}
    try:
        for dependent in (True, False):
            ctx.set_dependent_launch(dependent)
            plans, bufs = [], [torch.from_numpy(a).cuda()]
            for k, n, b, bias, mult, shift in layers:
                desc, keep = capi.make_gemm_desc(M, n, k, capi.U8, capi.S8, capi.U8, -2, 0, multipliers=mult, shifts=shift,
                                                 offset=4, min_bound=0, max_bound=255, has_bias=True)
                plan = capi.GemmPlan(ctx, desc, keep)
                plan.prepare(torch.from_numpy(b.view(np.uint8)).cuda())
                plans.append((plan, torch.from_numpy(bias).cuda()))
                bufs.append(torch.zeros((M, n), dtype=torch.uint8, device="cuda"))
            for _ in range(20):
                for i, (plan, d_bias) in enumerate(plans):
                    plan.run(bufs[i], None, d_bias, bufs[i + 1])
            ctx.sync()
            results[dependent] = bufs[-1].cpu().numpy()
            for plan, _ in plans:
                plan.close()
    finally:
        ctx.set_dependent_launch(True)
    assert np.array_equal(results[True], want)
    assert np.array_equal(results[False], want)
