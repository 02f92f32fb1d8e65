"""What the quantized linear path is timed on: the calls a serving program makes, through the layers and operators
that it uses, over the row counts, layer shapes and weight formats that this package takes.

Kinds of case
  linear   one quantized projection, called as a layer is called: GPTQ (4 / 8 bit, with and without act-order) and AWQ
           layers, fp8, NVFP4 / MXFP4 and HQQ weights through their apply functions
  moe      one mixture-of-experts layer (routing given): alignment, gate_up, SiLU, down, sum over the experts
  block    the linear part of one decoder block as a decode loop runs it: captured once in a CUDA graph, replayed
  repack   checkpoint layout -> kernel layout of one layer's weights, what loading a model spends its time on
"""
import math

import torch

from vllm_b200 import _custom_ops as ops
from vllm_b200.fused_moe import fused_marlin_moe
from vllm_b200.linear import ColumnParallelLinear
from vllm_b200.marlin_utils import marlin_make_workspace_new, marlin_permute_scales
from vllm_b200.marlin_utils_fp4 import apply_fp4_marlin_linear, prepare_fp4_layer_for_marlin
from vllm_b200.marlin_utils_fp8 import apply_fp8_marlin_linear, prepare_fp8_layer_for_marlin
from vllm_b200.quantization import AWQMarlinConfig, GPTQMarlinConfig
from vllm_b200.scalar_type import scalar_types

DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
EXPERTS, TOP_K = 8, 2
MOST_FLOPS = 2.0 * 4096 * 4096 * 28672   # the largest listed case's


def _linear(name, fmt, m, k, n, dtype="bf16", group=128, act_order=False, bias=False):
    c = {"kind": "linear", "format": fmt, "m": m, "k": k, "n": n, "dtype": dtype, "group": group,
         "act_order": act_order, "bias": bias}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one new token of one sequence through the attention projection of an 8B-sized model with
        # act-order GPTQ weights; latency and launches are what counts
        _linear("qkv_1", "gptq4", 1, 4096, 6144, act_order=True),
        # a handful of sequences, AWQ weights (zero-points), fp16, with the bias that some models have here
        _linear("awq_qkv_7", "awq4", 7, 3584, 4608, dtype="fp16", bias=True),
        # the widest projection of the block for 16 sequences
        _linear("gate_up_16", "gptq4", 16, 4096, 28672, act_order=True),
        # a larger decode batch, deep and narrow projection
        _linear("down_48", "gptq4", 48, 14336, 4096),
        # one token each of 24 sequences, fp8 weights with a scale per column
        _linear("fp8_gate_up_24", "fp8", 24, 4096, 28672, group=-1),
        # a short prompt (or a chunk of one) of a ragged length, 8-bit weights with a scale per column
        _linear("w8_gate_up_333", "gptq8", 333, 3584, 37888, dtype="fp16", group=-1),
        # a chunk of about a thousand prompt tokens, NVFP4 weights
        _linear("nvfp4_gate_up_1000", "nvfp4", 1000, 4096, 28672, group=16),
        # the largest call: 4096 prompt tokens through the widest projection
        _linear("gate_up_4096", "gptq4", 4096, 4096, 28672),
        # decode of 16 sequences and a 500-token prompt through a mixture-of-experts layer
        {"kind": "moe", "name": "moe_16", "format": "gptq4", "m": 16, "k": 4096, "n": 14336, "dtype": "bf16", "group": 128},
        {"kind": "moe", "name": "moe_500", "format": "gptq4", "m": 500, "k": 4096, "n": 14336, "dtype": "bf16", "group": 128},
        # one decode step of four sequences through the projections and norms of one block, as a replayed graph
        {"kind": "block", "name": "block_4", "m": 4, "hidden": 4096, "qkv": 6144, "inter": 14336, "dtype": "bf16"},
        # loading: the widest projection's weights with the rows in act-order
        {"kind": "repack", "name": "repack_gate_up", "format": "gptq4", "k": 4096, "n": 28672, "act_order": True},
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["linear"] * 9 + ["moe", "moe", "block", "repack"])
    if kind == "repack":
        return {"kind": "repack", "format": rng.choice(["gptq4", "gptq8", "awq4"]), "k": _log_int(rng, 1024, 14336, 128),
                "n": _log_int(rng, 1024, 28672, 64), "act_order": rng.random() < 0.5}
    if kind == "block":
        hidden = _log_int(rng, 1024, 8192, 128)
        return {"kind": "block", "m": _log_int(rng, 1, 64), "hidden": hidden, "qkv": hidden + 2 * _log_int(rng, 256, 2048, 64),
                "inter": _log_int(rng, 2048, 14336, 128), "dtype": rng.choice(["bf16", "fp16"])}
    if kind == "moe":
        return {"kind": "moe", "format": rng.choice(["gptq4", "gptq4", "gptq8", "awq4"]), "m": _log_int(rng, 1, 1024),
                "k": _log_int(rng, 1024, 4096, 128), "n": _log_int(rng, 1024, 14336, 128),
                "dtype": rng.choice(["bf16", "fp16"]), "group": rng.choice([128, 64])}
    fmt = rng.choice(["gptq4"] * 4 + ["gptq8", "gptq8", "awq4", "awq4", "fp8", "fp8", "nvfp4", "nvfp4", "mxfp4", "hqq4"])
    dtype = {"mxfp4": "bf16", "hqq4": "fp16"}.get(fmt) or rng.choice(["bf16", "fp16"])
    group = {"nvfp4": 16, "mxfp4": 32, "hqq4": 64}.get(fmt) or rng.choice([-1, 32, 64, 128, 128, 128])
    act_order = fmt == "gptq4" and group != -1 and rng.random() < 0.5
    m, k, n = _log_int(rng, 1, 4096), _log_int(rng, 1024, 14336, 128), _log_int(rng, 1024, 28672, 64)
    while 2.0 * m * k * n > MOST_FLOPS:
        n = _log_int(rng, 1024, 28672, 64)
        m = _log_int(rng, 1, 4096)
    return _linear(None, fmt, m, k, n, dtype=dtype, group=group, act_order=act_order, bias=rng.random() < 0.25)


# ---- inputs -----------------------------------------------------------------------------------------------------------


class _Plain(torch.nn.Module):
    """A layer whose attributes the preparation functions fill in."""


def _words(gen, *shape):
    """Packed codes: all values of the codes are met."""
    return torch.randint(-2**31, 2**31 - 1, shape, dtype=torch.int32, device=DEVICE, generator=gen)


def _scales(gen, dtype, *shape):
    return (torch.rand(shape, device=DEVICE, generator=gen) * 0.018 + 0.002).to(dtype)


def _checkpoint_layer(gen, fmt, k, n, dtype, group, act_order=False, bias=False):
    """A GPTQ / AWQ layer with random checkpoint tensors, loaded the way a model loads it."""
    if fmt == "awq4":
        config = AWQMarlinConfig(4, group)
    else:
        config = GPTQMarlinConfig(8 if fmt == "gptq8" else 4, group, desc_act=act_order)
    layer = ColumnParallelLinear(k, n, bias=bias, quant_config=config, params_dtype=dtype, device=DEVICE)
    layer.qweight.data.copy_(_words(gen, *layer.qweight.shape))
    layer.scales.data.copy_(_scales(gen, dtype, *layer.scales.shape))
    if fmt == "awq4":
        layer.qzeros.data.copy_(_words(gen, *layer.qzeros.shape))
    elif act_order:
        groups = torch.arange(k, device=DEVICE) // group
        layer.g_idx.data.copy_(groups[torch.randperm(k, device=DEVICE, generator=gen)])
    if bias:
        layer.bias.data.copy_(torch.randn(n, device=DEVICE, generator=gen))
    layer.process_weights_after_loading()
    return layer


def _float_layer(gen, fmt, k, n, dtype, group, bias):
    """fp8 / fp4 / HQQ weights; returns a function of the activations."""
    layer = _Plain()
    layer.input_size_per_partition, layer.output_size_per_partition = k, n
    b = torch.randn(n, device=DEVICE, generator=gen).to(dtype) if bias else None
    if fmt == "fp8":
        layer.orig_dtype = dtype
        layer.weight = (torch.randn(n, k, device=DEVICE, generator=gen) * 100).clamp(-448, 448).to(torch.float8_e4m3fn)
        layer.weight_scale = torch.rand((n,) if group == -1 else (n, k // group), device=DEVICE, generator=gen) * 4e-4 + 1e-4
        prepare_fp8_layer_for_marlin(layer, size_k_first=False)
        return lambda x: apply_fp8_marlin_linear(x, layer.weight, layer.weight_scale, layer.workspace, n, k, b)
    if fmt in ("nvfp4", "mxfp4"):
        layer.params_dtype = dtype
        layer.weight = torch.nn.Parameter(torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device=DEVICE,
                                                        generator=gen), requires_grad=False)
        if fmt == "nvfp4":
            scale = (torch.rand(n, k // 16, device=DEVICE, generator=gen) * 400 + 20).to(torch.float8_e4m3fn)
            layer.weight_scale_2 = torch.nn.Parameter(torch.rand(1, device=DEVICE, generator=gen) * 2e-5 + 4e-5,
                                                      requires_grad=False)
        else:
            scale = torch.randint(117, 122, (n, k // 32), dtype=torch.uint8, device=DEVICE, generator=gen)
        layer.weight_scale = torch.nn.Parameter(scale, requires_grad=False)
        layer.bias = torch.nn.Parameter(b, requires_grad=False) if bias else None
        prepare_fp4_layer_for_marlin(layer)
        return lambda x: apply_fp4_marlin_linear(x, layer.weight, layer.weight_scale, getattr(layer, "weight_scale_2", None),
                                                 layer.workspace, n, k, layer.bias)
    q = _words(gen, k // 16, 2 * n)
    s = marlin_permute_scales(_scales(gen, dtype, k // group, n), k, n, group)
    z = marlin_permute_scales((8 + torch.randn(k // group, n, device=DEVICE, generator=gen)).to(dtype), k, n, group)
    ws = marlin_make_workspace_new(torch.device(DEVICE))
    return lambda x: ops.gptq_marlin_gemm(x, None, q, b, s, None, z, None, None, ws, scalar_types.uint4, x.shape[0], n, k,
                                          is_k_full=True, use_fp32_reduce=True, is_zp_float=True)


def _moe(gen, c, dtype):
    """Weights of all experts in kernel layout; the router's choice for every token."""
    bits = 8 if c["format"] == "gptq8" else 4
    m, k, n, g = c["m"], c["k"], c["n"], c["group"]
    args = {"hidden_states": torch.randn(m, k, device=DEVICE, generator=gen).to(dtype),
            "w1": _words(gen, EXPERTS, k // 16, 2 * n * bits // 2), "w2": _words(gen, EXPERTS, n // 16, k * bits // 2),
            "w1_scale": _scales(gen, dtype, EXPERTS, k // g, 2 * n), "w2_scale": _scales(gen, dtype, EXPERTS, n // g, k)}
    if bits == 8:   # codes reach 16 times further
        args["w1_scale"] /= 16
        args["w2_scale"] /= 16
    args["quant_type"] = {"gptq4": scalar_types.uint4b8, "gptq8": scalar_types.uint8b128, "awq4": scalar_types.uint4}[c["format"]]
    if c["format"] == "awq4":
        args["w1_zeros"] = _words(gen, EXPERTS, k // g, 2 * n // 8)
        args["w2_zeros"] = _words(gen, EXPERTS, n // g, k // 8)
    router = torch.softmax(torch.randn(m, EXPERTS, device=DEVICE, generator=gen), dim=-1)
    weights, ids = torch.topk(router, TOP_K, dim=-1)
    args["topk_weights"], args["topk_ids"] = weights.contiguous(), ids.to(torch.int32).contiguous()
    args["workspace"] = marlin_make_workspace_new(torch.device(DEVICE))
    return args


class _Block:
    """Projections and norms of one decoder block.  Attention is another library's kernel: the query columns stand in
    for its output."""

    def __init__(self, gen, c, dtype):
        h, inter = c["hidden"], c["inter"]
        make = lambda k, n: _checkpoint_layer(gen, "gptq4", k, n, dtype, 128)  # noqa: E731
        self.qkv, self.o, self.gate_up, self.down = make(h, c["qkv"]), make(h, h), make(h, 2 * inter), make(inter, h)
        self.norms = [(1 + 0.1 * torch.randn(h, device=DEVICE, generator=gen)).to(dtype) for _ in range(3)]
        self.x = torch.randn(c["m"], h, device=DEVICE, generator=gen).to(dtype)
        self.step()                                    # once outside the capture, as a program does
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.out = self.step()

    def step(self):
        residual = self.x.clone()
        h = torch.empty_like(residual)
        ops.rms_norm(h, residual, self.norms[0], 1e-5)
        attn = self.qkv(h)[:, :h.shape[1]]
        h = self.o(attn)
        ops.fused_add_rms_norm(h, residual, self.norms[1], 1e-5)
        gu = self.gate_up(h)
        act = torch.empty(gu.shape[0], gu.shape[1] // 2, dtype=gu.dtype, device=gu.device)
        ops.silu_and_mul(act, gu)
        h = self.down(act)
        ops.fused_add_rms_norm(h, residual, self.norms[2], 1e-5)
        return h, residual


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    kind, dtype = case["kind"], DTYPES[case.get("dtype", "bf16")]
    if kind == "block":
        return {"kind": kind, "block": _Block(gen, case, dtype)}
    if kind == "moe":
        return {"kind": kind, "args": _moe(gen, case, dtype)}
    k, n = case["k"], case["n"]
    if kind == "repack":
        bits = 8 if case["format"] == "gptq8" else 4
        if case["format"] == "awq4":
            return {"kind": "repack_awq", "args": (_words(gen, k, n * bits // 32), k, n, bits)}
        perm = torch.empty(0, dtype=torch.int32, device=DEVICE)
        if case["act_order"]:
            perm = torch.randperm(k, device=DEVICE, generator=gen).to(torch.int32)
        return {"kind": "repack_gptq", "args": (_words(gen, k * bits // 32, n), perm, k, n, bits)}
    if case["format"] in ("gptq4", "gptq8", "awq4"):
        layer = _checkpoint_layer(gen, case["format"], k, n, dtype, case["group"], case["act_order"], case["bias"])
    else:
        layer = _float_layer(gen, case["format"], k, n, dtype, case["group"], case["bias"])
    return {"kind": kind, "layer": layer, "x": torch.randn(case["m"], k, device=DEVICE, generator=gen).to(dtype)}


# ---- one pass ---------------------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "moe":
        return fused_marlin_moe(**state["args"])
    if kind == "block":
        state["block"].graph.replay()
        return state["block"].out
    if kind == "repack_awq":
        return ops.awq_marlin_repack(*state["args"])
    return ops.gptq_marlin_repack(*state["args"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------


def _weight_bytes(fmt, k, n, group):
    bits = 8 if fmt in ("gptq8", "fp8") else 4
    groups = 1 if group == -1 else k // group
    scale = 1 if fmt in ("nvfp4", "mxfp4") else 2
    zeros = {"awq4": groups * n * bits // 8, "hqq4": groups * n * 2}.get(fmt, 0)
    return k * n * bits // 8 + groups * n * scale + zeros


def work(case):
    kind = case["kind"]
    if kind == "repack":
        bits = 8 if case["format"] == "gptq8" else 4
        perm = 4 * case["k"] if case["act_order"] and case["format"] != "awq4" else 0
        return {"bytes": 2 * case["k"] * case["n"] * bits // 8 + perm, "flops": 0}
    m = case["m"]
    if kind == "block":
        h, qkv, inter = case["hidden"], case["qkv"], case["inter"]
        shapes = [(h, qkv), (h, h), (h, 2 * inter), (inter, h)]
        return {"bytes": sum(_weight_bytes("gptq4", k, n, 128) for k, n in shapes) + 6 * m * h + 6 * h,
                "flops": sum(2 * m * k * n for k, n in shapes)}
    k, n = case["k"], case["n"]
    if kind == "moe":
        used = min(EXPERTS, m * TOP_K)
        per_expert = _weight_bytes(case["format"], k, 2 * n, case["group"]) + _weight_bytes(case["format"], n, k, case["group"])
        return {"bytes": used * per_expert + 4 * m * k + 8 * m * TOP_K, "flops": 2 * m * TOP_K * 3 * k * n}
    index = 8 * k if case["act_order"] else 0
    return {"bytes": _weight_bytes(case["format"], k, n, case["group"]) + index + 2 * m * k + 2 * m * n + (2 * n if case["bias"] else 0),
            "flops": 2 * m * k * n}


def tolerance(case):
    if case["kind"] == "repack":
        return "exact"
    # a 16-bit rounding of the result, and of the scaled weights where a kernel rounds them before the product
    if case["kind"] == "linear":
        return {"rel": 2e-3} if case["dtype"] == "fp16" else {"rel": 1e-2}
    return {"rel": 4e-3} if case["dtype"] == "fp16" else {"rel": 1.5e-2}
