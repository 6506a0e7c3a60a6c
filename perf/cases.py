"""The work a user of this library has it do, as timed cases.

Every case goes through the public Python binding (``computelibrary_b200``): a configured ``GemmPlan`` /
``ConvPlan`` or a captured ``ResNet50`` is what a program keeps, ``run`` is one call on device-resident
operands.  All results are integers, or floats produced by one conversion and one multiplication, and the
arithmetic contract is bit-exact, so every tolerance is "exact".
"""
from __future__ import annotations

import math

import numpy as np
import torch

import computelibrary_b200 as cl
from computelibrary_b200 import capi, resnet50

DTYPE = {"u8": capi.U8, "s8": capi.S8, "s32": capi.S32, "f32": capi.F32}
TORCH = {"u8": torch.uint8, "s8": torch.int8, "s32": torch.int32, "f32": torch.float32}
DST_BYTES = {"u8": 1, "s8": 1, "s32": 4, "f32": 4}
MACS_MAX = 8192 * 14336 * 4096  # the largest listed product: nothing drawn costs more


# ---- cases ------------------------------------------------------------------------------------------------
def gemm(M, N, K, a="s8", b="s8", out="s8", per_channel=True, bias=True, **more):
    """A fused GEMMLowp on constant weights.  u8 weights are asymmetric (per-tensor scale, zero point)."""
    return dict(kind="gemm", M=M, N=N, K=K, a=a, b=b, out=out, per_channel=per_channel, bias=bias, **more)


def batched(batch, M, N, K, a="u8", b="u8", out="u8"):
    """A batch of products whose B operand changes with every call (both operands are activations)."""
    return dict(kind="batched", batch=batch, M=M, N=N, K=K, a=a, b=b, out=out)


def two_stage(M, N, K):
    """NEGEMMLowpMatrixMultiplyCore to S32 followed by a stand-alone NEGEMMLowpOutputStage."""
    return dict(kind="two_stage", M=M, N=N, K=K)


def conv(B, H, C, OFM, k, stride, w="s8", zero_point=128):
    """NHWC convolution, square image and kernel, padding k // 2.  w: s8 = per-channel symmetric weights,
    u8 = per-tensor weights with a zero point."""
    return dict(kind="conv", B=B, H=H, C=C, OFM=OFM, k=k, stride=stride, w=w, zero_point=zero_point)


def resnet(batch):
    return dict(kind="resnet50", batch=batch)


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # the smallest call: examples/neon_gemm_qasymm8 sizes, both operands asymmetric; latency is all it has
        named("gemm_small", gemm(64, 128, 256, "u8", "u8", "u8", per_channel=False)),
        # odd sizes in every direction (the validation suite's large GEMMLowp shapes): unaligned rows of A and dst
        named("gemm_ragged", gemm(923, 429, 873, "u8", "u8", "u8", per_channel=False)),
        # the square product of the benchmark
        named("gemm_square", gemm(4096, 4096, 4096)),
        # a transformer's wide linear layer: a prompt of 8192 tokens (the largest case), and token-by-token decoding
        # of 16 sequences with the same weights
        named("linear_prefill", gemm(8192, 14336, 4096, bias=False)),
        named("linear_decode", gemm(16, 14336, 4096, bias=False)),
        # the same kind of layer handing float32 to an unquantized consumer, at an ordinary number of tokens
        named("linear_f32", gemm(512, 4096, 4096, out="f32", per_channel=False, bias=False)),
        # products of activations with activations: B is re-laid out by every call
        named("batched_dynamic", batched(16, 384, 384, 128)),
        # an S32 product and the output stage as two functions (programs written against the unfused API)
        named("two_stage", two_stage(1024, 1024, 1024)),
        # a quantized 3x3 layer with per-channel weights and a non-zero input zero point, batch 32
        named("conv3x3", conv(32, 56, 64, 64, 3, 1)),
        # a 3x3 layer of a per-tensor QASYMM8 network (asymmetric weights)
        named("conv3x3_asymmetric", conv(32, 28, 128, 128, 3, 1, w="u8")),
        # image classification, one image at a time and at the batch of the benchmark
        named("resnet50_b1", resnet(1)),
        named("resnet50_b256", resnet(256)),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges; half of the sizes are whatever comes up, half are multiples of 16."""
    def size(lo, hi):
        v = _log(rng, lo, hi)
        return v if rng.random() < 0.5 or hi < 16 else max(16, v // 16 * 16)

    kind = rng.choice(["gemm", "gemm", "gemm", "batched", "two_stage", "conv", "conv", "resnet50"])
    if kind == "gemm":
        while True:
            M, N, K = size(1, 8192), size(64, 14336), size(64, 8192)
            if M * N * K <= MACS_MAX:
                break
        a, b, per_channel = rng.choice([("s8", "s8", True), ("u8", "s8", True), ("u8", "u8", False)])
        out = rng.choice([a, a, a, "f32"])
        return gemm(M, N, K, a, b, out, per_channel and out != "f32", out != "f32" and rng.random() < 0.5)
    if kind == "batched":
        t = rng.choice(["u8", "s8"])
        return batched(rng.randint(2, 32), size(16, 1024), size(16, 1024), size(16, 512), t, t, t)
    if kind == "two_stage":
        return two_stage(size(16, 4096), size(16, 4096), size(64, 4096))
    if kind == "conv":
        k = rng.choice([1, 3, 3, 5])
        C, OFM = size(16, 512), size(16, 512)
        return conv(_log(rng, 1, 64), rng.randint(7, 64), C, OFM, k, rng.choice([1, 1, 2]), rng.choice(["s8", "s8", "u8"]),
                    rng.choice([0, 128]))
    return resnet(_log(rng, 1, 256))


# ---- inputs -----------------------------------------------------------------------------------------------
class _Draw:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.rng = np.random.default_rng(seed)

    def q8(self, shape, kind, lo=None, hi=None):
        info = torch.iinfo(TORCH[kind])
        lo, hi = info.min if lo is None else lo, info.max if hi is None else hi
        return torch.randint(lo, hi + 1, shape, dtype=TORCH[kind], device="cuda", generator=self.gen)

    def activations(self, shape, kind):
        """Clipped Gaussian codes around the middle of the type, as calibrated activations are."""
        info = torch.iinfo(TORCH[kind])
        mid = 128.0 if kind == "u8" else 0.0
        v = torch.empty(shape, dtype=torch.float16, device="cuda").normal_(0.0, 30.0, generator=self.gen)
        return (v + mid).round_().clamp_(info.min, info.max).to(TORCH[kind])

    def bias(self, n, k):
        r = int(30 * 73 * math.sqrt(k))
        return torch.randint(-r, r + 1, (n,), dtype=torch.int32, device="cuda", generator=self.gen)


def _real_multiplier(k):
    """Maps sums of K products (activation spread 30, uniform weights) to a spread of about 40 output codes."""
    return 40.0 / (30.0 * 73.0 * math.sqrt(k))


def _stage(d, k, n, per_channel):
    if not per_channel:
        m, s = capi.calculate_quantized_multiplier(np.float32(_real_multiplier(k)))
        return dict(multiplier=m, shift=s)
    spread = np.exp(d.rng.uniform(np.log(0.3), np.log(3.0), n)).astype(np.float32)
    m, s = capi.calculate_quantized_multipliers(np.float32(1.0), (spread * np.float32(_real_multiplier(k))).astype(np.float32),
                                                np.float32(1.0))
    return dict(multipliers=m, shifts=s)


def _zero_point(kind):
    return 128 if kind == "u8" else -5


def prepare(case, seed):
    d = _Draw(seed)
    st = dict(case=case)
    kind = case["kind"]
    if kind == "resnet50":
        st["stream"] = torch.cuda.Stream()
        st["ctx"] = ctx = cl.Context(torch.cuda.current_device(), st["stream"].cuda_stream)
        nodes = resnet50.build_graph()
        params = resnet50.synthetic_params(nodes, seed=seed % 100003, fan_in_scaled=True)
        st["net"] = resnet50.ResNet50(ctx, case["batch"], params=params, nodes=nodes)
        st["images"] = d.q8((case["batch"], 224, 224, 3), "u8")
        torch.cuda.current_stream().synchronize()
        st["graph"] = st["net"].capture(st["images"], st["stream"])
        return st
    st["ctx"] = ctx = cl.Context(torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream)
    if kind == "conv":
        B, H, C, OFM, k = (case[x] for x in ("B", "H", "C", "OFM", "k"))
        wzp = 120 if case["w"] == "u8" else 0
        desc, keep = capi.make_conv_desc(
            B, H, H, C, OFM, k, k, (case["stride"],) * 2, (k // 2,) * 4, (1, 1), capi.U8, DTYPE[case["w"]], case["zero_point"], wzp,
            dst_zp=case["zero_point"], min_bound=case["zero_point"], max_bound=255, has_bias=True,
            **_stage(d, k * k * C, OFM, case["w"] == "s8"))
        st["plan"] = plan = cl.ConvPlan(ctx, desc, keep)
        wo, ho = plan.out_dims()
        st["src"] = d.activations((B, H, H, C), "u8")
        st["bias"] = d.bias(OFM, k * k * C)
        st["dst"] = torch.empty((B, ho, wo, OFM), dtype=torch.uint8, device="cuda")
        lo = {} if case["w"] == "u8" else dict(lo=-127)
        plan.prepare(d.q8((OFM, k, k, C), case["w"], **lo))
        ctx.sync()
        return st
    M, N, K = case["M"], case["N"], case["K"]
    if kind == "two_stage":
        a, b, out, batch, stage = "u8", "u8", "s32", 1, capi.STAGE_NONE
    else:
        a, b, out, batch = case["a"], case["b"], case["out"], case.get("batch", 1)
        stage = capi.STAGE_NONE if out == "f32" else capi.STAGE_FIXEDPOINT
    more = {}
    if stage == capi.STAGE_FIXEDPOINT:
        info = torch.iinfo(TORCH[out])
        more = dict(_stage(d, K, N, case.get("per_channel", False)), offset=128 if out == "u8" else 0, min_bound=info.min, max_bound=info.max,
                    has_bias=bool(case.get("bias", False)))
    elif out == "f32":
        more = dict(dequantize_scale=0.02 * 0.005)
    desc, keep = capi.make_gemm_desc(
        M, N, K, DTYPE[a], DTYPE[b], DTYPE[out], -_zero_point(a), -120 if b == "u8" else 0, stage, batch=batch,
        b_batch_stride=K * N if batch > 1 else 0, b_constant=kind != "batched", **more)
    st["plan"] = plan = cl.GemmPlan(ctx, desc, keep)
    lead = (batch,) if batch > 1 else ()
    st["a"] = d.activations(lead + (M, K), a)
    weights = d.activations(lead + (K, N), b) if kind == "batched" else d.q8((K, N), b, **({} if b == "u8" else dict(lo=-127)))
    st["bias"] = d.bias(N, K) if more.get("has_bias") or kind == "two_stage" else None
    st["dst"] = torch.empty(lead + (M, N), dtype=TORCH[out], device="cuda")
    if kind == "batched":
        st["b"] = weights
    else:
        plan.prepare(weights)
    if kind == "two_stage":
        st["q"] = torch.empty((M, N), dtype=torch.uint8, device="cuda")
        st["mult"], st["shift"] = capi.calculate_quantized_multiplier(np.float32(_real_multiplier(K)))
    ctx.sync()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "resnet50":
        st["graph"].replay()
        return {"logits": st["net"].bufs["logits"], "classes": st["net"].bufs["softmax"]}
    if kind == "conv":
        st["plan"].run(st["src"], st["bias"], st["dst"])
        return st["dst"]
    if kind == "batched":
        st["plan"].run(st["a"], st["b"], None, st["dst"])
        return st["dst"]
    if kind == "two_stage":
        st["plan"].run(st["a"], None, None, st["dst"])
        M, N = case["M"], case["N"]
        st["ctx"].output_stage(st["dst"], 4 * N, st["bias"], st["q"], N, capi.U8, M, N, None, None, st["mult"], st["shift"], 1, 128, 0, 255)
        return {"s32": st["dst"], "u8": st["q"]}
    st["plan"].run(st["a"], None, st["bias"], st["dst"])
    return st["dst"]


# ---- what a pass cannot do without ------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "resnet50":
        nodes = resnet50.build_graph()
        B = case["batch"]
        weights = sum(n["ofm"] * (n["k"] ** 2 * n["in_shape"][2] + 12) for n in nodes if n["op"] == "conv")
        return {"bytes": B * (224 * 224 * 3 + 2 * 1000) + weights, "flops": B * resnet50.graph_ops(nodes)}
    if kind == "conv":
        B, H, C, OFM, k, s = (case[x] for x in ("B", "H", "C", "OFM", "k", "stride"))
        o = (H + 2 * (k // 2) - k) // s + 1
        return {"bytes": B * H * H * C + k * k * C * OFM + 4 * OFM + B * o * o * OFM, "flops": 2.0 * B * o * o * OFM * k * k * C}
    M, N, K, batch = case["M"], case["N"], case["K"], case.get("batch", 1)
    out = 5 if kind == "two_stage" else DST_BYTES[case["out"]]
    return {"bytes": batch * (M * K + K * N + M * N * out) + 4 * N, "flops": 2.0 * batch * M * N * K}


def tolerance(case):
    """Integer results with a bit-exact contract; the float32 results are one rounding of an exact integer and one
    multiplication, the softmax one fixed evaluation order of expf."""
    return "exact"
