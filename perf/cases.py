"""Performance cases of the quantized linear path.

A case is a run of decoder layers as a serving engine drives them: per layer the four
projections qkv -> o -> gate_up -> down, through the tensor-parallel layer classes (one rank)
or, on the fused route, through the producers that quantise their own output.  What varies:

* ``scheme``   "w8a8" (int8 weights, activations quantised per token) or "int8" (W8A16);
* ``tokens``   1 (one sequence decoding) to 16384 (a full prefill batch);
* ``hidden``, ``q``, ``kv``, ``inter``  widths of the model (or of one rank's share of it):
  qkv is hidden -> q + 2 kv, o is q -> hidden, gate_up is hidden -> 2 inter, down is
  inter -> hidden.  The listed ones are the Qwen3-0.6B and Qwen3-8B architectures that the
  benchmark uses and one rank of the latter at TP = 8;
* ``layers``   how many layers, each with weights of its own.  Decode runs enough of them that
  the weights come from HBM, as they do in a whole model;
* ``launch``   "eager" (prefill always; decode with ``enforce_eager``) or "graph" (decode: one
  captured CUDA graph per batch size, replayed every step);
* ``route``    "plain": every layer object is called on a 16-bit tensor; "fused": RMSNorm with
  the residual add and SiLU-mul hand int8 codes to the next projection (W8A8 only);
* ``dtype``    "bf16" or "fp16"; ``bias``  whether the projections have one.

Attention is the caller's business: its output is an input of the case.
"""
import math

import torch

from tiny_vllm_b200.layers.linear import (MergedColumnParallelLinear, QKVParallelLinear,
                                          RowParallelLinear)
from tiny_vllm_b200.quantization.cuda import add_rmsnorm_quantize_int8, silu_mul_quantize_int8
from tiny_vllm_b200.quantization.utils import quantize_int8_per_channel

HEAD = 128
EPS = 1e-6
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

QWEN3_0_6B = {"hidden": 1024, "q": 2048, "kv": 1024, "inter": 3072}
QWEN3_8B = {"hidden": 4096, "q": 4096, "kv": 1024, "inter": 12288}
QWEN3_8B_TP8 = {"hidden": 4096, "q": 512, "kv": 128, "inter": 1536}

# Cost limits of a drawn case: the largest listed one (16384 tokens through a layer of the 8B
# model) and the largest set of weights.
MAX_MACS = 16384 * 192_937_984
MAX_WEIGHT_BYTES = 4 * 192_937_984


def _case(name, scheme, tokens, model, layers, launch, route="plain", dtype="bf16", bias=False):
    return {"name": name, "scheme": scheme, "tokens": tokens, **model, "layers": layers,
            "launch": launch, "route": route, "dtype": dtype, "bias": bias}


def listed():
    return [
        # one sequence decoding without CUDA graphs: the smallest calls, one launch after another
        _case("w8a8 0.6b decode 1 eager", "w8a8", 1, QWEN3_0_6B, 4, "eager"),
        # a short prompt joining a batch: prefill is always eager, its length is anything; a
        # model family with fp16 weights and biased projections
        _case("w8a16 0.6b prefill 77 fp16", "int8", 77, QWEN3_0_6B, 2, "eager", dtype="fp16",
              bias=True),
        # decode steps from captured graphs: few sequences, many, and a full batch
        _case("w8a16 0.6b decode 16 graph", "int8", 16, QWEN3_0_6B, 12, "graph"),
        _case("w8a8 0.6b decode 256 graph", "w8a8", 256, QWEN3_0_6B, 12, "graph"),
        _case("w8a16 0.6b decode 512 graph", "int8", 512, QWEN3_0_6B, 12, "graph"),
        # the larger model: one interactive user, a small batch, and a TP = 8 rank's share
        _case("w8a16 8b decode 1 graph", "int8", 1, QWEN3_8B, 4, "graph"),
        _case("w8a8 8b decode 32 graph", "w8a8", 32, QWEN3_8B, 4, "graph"),
        _case("w8a16 8b/tp8 decode 64 graph", "int8", 64, QWEN3_8B_TP8, 8, "graph"),
        # prefill batches: several prompts of odd total length on the fused producers, the
        # benchmark's 8192 tokens, a W8A16 batch of the larger model, the engine's largest batch
        _case("w8a8 0.6b prefill 1999 fused", "w8a8", 1999, QWEN3_0_6B, 2, "eager", route="fused"),
        _case("w8a8 0.6b prefill 8192", "w8a8", 8192, QWEN3_0_6B, 1, "eager"),
        _case("w8a16 8b prefill 3000", "int8", 3000, QWEN3_8B, 1, "eager"),
        _case("w8a8 8b prefill 16384", "w8a8", 16384, QWEN3_8B, 1, "eager"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    scheme = rng.choice(("w8a8", "int8"))
    launch = rng.choice(("eager", "graph"))
    route = "fused" if scheme == "w8a8" and rng.random() < 0.3 else "plain"
    hidden = 64 * round(_log_uniform(rng, 1024, 4096) / 64)
    # query width: from one rank's share of a tensor-parallel model to twice the hidden size
    q = HEAD * max(1, round(_log_uniform(rng, hidden / 8, 2 * hidden) / HEAD))
    kv = HEAD * max(1, round(q / HEAD / rng.choice((1, 2, 4, 8))))
    inter = 32 * round(_log_uniform(rng, 3 * hidden / 8, 3 * hidden) / 32)
    per_layer = hidden * (q + 2 * kv) + q * hidden + hidden * 2 * inter + inter * hidden
    tokens = round(_log_uniform(rng, 1, 512 if launch == "graph" else 16384))
    tokens = max(1, min(tokens, MAX_MACS // per_layer))
    if launch == "graph":
        layers = 2 if route == "fused" else max(2, min(12, -(-192_000_000 // per_layer)))
    else:
        layers = 4 if tokens <= 64 else 2 if tokens <= 2048 else 1
    layers = max(1, min(layers, MAX_WEIGHT_BYTES // per_layer, MAX_MACS // (per_layer * tokens)))
    return {"scheme": scheme, "tokens": tokens, "hidden": hidden, "q": q, "kv": kv, "inter": inter,
            "layers": layers, "launch": launch, "route": route,
            "dtype": rng.choice(("bf16", "bf16", "fp16")), "bias": rng.random() < 0.2}


def _projections(case):
    """(in features, out features) of the four projections of a layer."""
    h, q, kv, inter = case["hidden"], case["q"], case["kv"], case["inter"]
    return (h, q + 2 * kv), (q, h), (h, 2 * inter), (inter, h)


def _activation(gen, tokens, width, dtype):
    """N(0, 1) with 1 % outlier channels scaled by 20."""
    x = torch.randn(tokens, width, device="cuda", generator=gen)
    outliers = torch.randperm(width, device="cuda", generator=gen)[: max(1, width // 100)]
    x[:, outliers] *= 20.0
    return x.to(dtype)


def _fill(layer, gen, dtype):
    """Weights N(0, 0.02) quantised per output channel, through the layer's loader hooks."""
    n, k = layer.qweight.shape
    codes, scales = quantize_int8_per_channel(
        torch.randn(n, k, device="cuda", generator=gen).mul_(0.02))
    layer.qweight.weight_loader(layer.qweight, codes)
    scale_param = layer.scales if hasattr(layer, "scales") else layer.w_scales
    scale_param.weight_loader(scale_param, scales)
    if layer.bias is not None:
        layer.bias.data.copy_(torch.randn(n, device="cuda", generator=gen).to(dtype))
    return layer


class _DecoderLinears:
    """The projections of one decoder layer and, on the fused route, its norm weights."""

    def __init__(self, case, gen, dtype):
        h, q, kv, inter = case["hidden"], case["q"], case["kv"], case["inter"]
        kw = {"bias": case["bias"], "quantization": case["scheme"]}
        before = torch.get_default_dtype()
        torch.set_default_dtype(dtype)
        try:
            with torch.device("cuda"):
                self.qkv = QKVParallelLinear(h, HEAD, q // HEAD, kv // HEAD, **kw)
                self.o = RowParallelLinear(q, h, **kw)
                self.gate_up = MergedColumnParallelLinear(h, [inter, inter], **kw)
                self.down = RowParallelLinear(inter, h, **kw)
        finally:
            torch.set_default_dtype(before)
        for layer in (self.qkv, self.o, self.gate_up, self.down):
            _fill(layer, gen, dtype)
        if case["route"] == "fused":
            self.norm1, self.norm2 = ((1 + 0.1 * torch.randn(h, device="cuda", generator=gen)).to(dtype)
                                      for _ in range(2))


class _State:
    pass


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    s = _State()
    s.dtype, s.fused, s.graph, s.out = dtype, case["route"] == "fused", None, None
    s.layers = [_DecoderLinears(case, gen, dtype) for _ in range(case["layers"])]
    m = case["tokens"]
    if s.fused:
        s.x = _activation(gen, m, case["hidden"], dtype)
        s.residual = _activation(gen, m, case["hidden"], dtype)
        s.attention = [_activation(gen, m, case["q"], dtype) for _ in s.layers]
    else:
        s.inputs = [[_activation(gen, m, k, dtype) for k, _ in _projections(case)]
                    for _ in s.layers]
    if case["launch"] == "graph":
        # as a model runner does it: one eager pass, then the capture
        with torch.inference_mode():
            _forward(s)
            s.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s.graph):
                s.out = _forward(s)
    return s


def _plain(s):
    out = []
    for layer, (x_qkv, x_o, x_gate_up, x_down) in zip(s.layers, s.inputs):
        out += [layer.qkv(x_qkv), layer.o(x_o), layer.gate_up(x_gate_up), layer.down(x_down)]
    return out


def _fused(s):
    x, residual, out = s.x, s.residual, []
    for layer, attention in zip(s.layers, s.attention):
        codes, scales, residual, _ = add_rmsnorm_quantize_int8(x, layer.norm1, EPS, residual)
        out.append(layer.qkv.quant_method.apply_quantized(codes, scales, layer.qkv, s.dtype))
        x = layer.o(attention)
        codes, scales, residual, _ = add_rmsnorm_quantize_int8(x, layer.norm2, EPS, residual)
        gate_up = layer.gate_up.quant_method.apply_quantized(codes, scales, layer.gate_up, s.dtype)
        codes, scales, _ = silu_mul_quantize_int8(gate_up)
        x = layer.down.quant_method.apply_quantized(codes, scales, layer.down, s.dtype)
    return out + [x, residual]


def _forward(s):
    return _fused(s) if s.fused else _plain(s)


def run(state):
    if state.graph is not None:
        state.graph.replay()
        return state.out
    with torch.inference_mode():
        return _forward(state)


def work(case):
    m, layers = case["tokens"], case["layers"]
    nbytes = flops = 0
    for k, n in _projections(case):
        nbytes += n * k + 4 * n + (2 * n if case["bias"] else 0)
        flops += 2 * m * n * k
        if case["route"] == "plain":
            nbytes += 2 * m * (k + n)
    if case["route"] == "fused":
        # per layer: attention output in, qkv out, two norm weights
        nbytes += 2 * m * (case["q"] + case["q"] + 2 * case["kv"]) + 4 * case["hidden"]
    nbytes, flops = layers * nbytes, layers * flops
    if case["route"] == "fused":
        nbytes += 4 * 2 * m * case["hidden"]    # x and residual, in and out
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["route"] == "fused":
        # a normalised value may round the other way and move an int8 code by one step
        return {"rel": 1e-2}
    if case["scheme"] == "w8a8":
        # int32 sums are exact, so are the codes: only the rounding of the result is left
        return {"rel": 2e-3 if case["dtype"] == "bf16" else 5e-4}
    # fp32 sums in another order, then the rounding of the result
    return {"rel": 4e-3 if case["dtype"] == "bf16" else 1e-3}
